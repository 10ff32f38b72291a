"""The inline assembly of the kernels, by reading its text: an output that an instruction writes before a later one of the same block
reads an input has to be early-clobber, or the compiler may give both the same register."""
import glob
import os
import re
import subprocess
import sys

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ditto_b200", "csrc")
STRING = r'"(?:[^"\\]|\\.)*"'


def _blocks(text):
    """(instructions, constraints of the outputs, number of operands) of every asm statement with outputs."""
    for m in re.finditer(r"\basm(?:\s+volatile)?\s*\(((?:\s*" + STRING + r")+)\s*:(?!:)((?:[^:\"]|" + STRING + r")*)(?::(?!:)((?:[^:\"]|" + STRING + r")*))?", text):
        code = "".join(s[1:-1] for s in re.findall(STRING, m.group(1))).replace("\\n", "").replace("\\t", "")
        outs = re.findall(STRING, m.group(2))
        ins = re.findall(STRING, m.group(3) or "")
        if outs:
            yield [c for c in code.split(";") if "%" in c.replace("%%", "")], [o[1:-1] for o in outs], len(outs) + len(ins)


def hazards(text):
    """Numbers of outputs that are written ahead of the last instruction with an input and are not early-clobber, per block."""
    found = []
    for code, outs, operands in _blocks(text):
        named = [{int(n) for n in re.findall(r"%(\d+)", c.replace("%%", ""))} for c in code]
        last = max((i for i, n in enumerate(named) if any(len(outs) <= o < operands for o in n)), default=-1)
        early = {o for n in named[:max(last, 0)] for o in n if o < len(outs) and "&" not in outs[o] and "+" not in outs[o]}
        if early:
            found.append((code[0].strip()[:60], sorted(early)))
    return found


def test_the_search_finds_one():
    plain = 'asm volatile("a %0, [%2];\\n\\t" "a %1, [%3];" : "=r"(x), "=r"(y) : "r"(p), "r"(q) : "memory");'
    assert hazards(plain) == [("a %0, [%2]", [0])]
    assert hazards(plain.replace('"=r"(x)', '"=&r"(x)')) == []
    assert hazards('asm("mov.b32 t, %2; cvt %0, t; cvt %1, t;" : "=f"(x), "=f"(y) : "r"(w));') == []


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_outputs_written_ahead_of_inputs(path):
    assert hazards(open(path).read()) == []


def test_generated_wrappers_are_the_generators():
    text = subprocess.run([sys.executable, os.path.join(CSRC, "gen_tmem_ops.py")], check=True, capture_output=True, text=True).stdout
    assert text == open(os.path.join(CSRC, "tmem_ops_gen.cuh")).read()
