"""Emit tmem_ops_gen.cuh: tcgen05.ld / tcgen05.st wrappers for the 32x32b shape.

Each wrapper moves N consecutive 32-bit TMEM columns of the calling thread's own
TMEM lane (lane = 32 * (warp_id % 4) + lane_id) to / from N registers.  The load
wrappers carry their `tcgen05.wait::ld` inside the same asm statement so the
compiler can never schedule a consumer of the registers before the wait.

Run:  python gen_tmem_ops.py > tmem_ops_gen.cuh
"""

def regs(n, start):
    return ", ".join(f"%{i}" for i in range(start, start + n))

def emit_ld(n):
    outs = ", ".join(f'"=r"(r[{i}])' for i in range(n))
    print(f"""__device__ __forceinline__ void tmem_ld_x{n}_wait(uint32_t taddr, uint32_t (&r)[{n}]) {{
  asm volatile(
    "tcgen05.ld.sync.aligned.32x32b.x{n}.b32 {{{regs(n, 0)}}}, [%{n}];\\n\\t"
    "tcgen05.wait::ld.sync.aligned;\\n"
    : {outs}
    : "r"(taddr) : "memory");
}}
""")

def emit_ld_2x32():
    # early-clobber: the first load writes its registers before the second one reads its address
    outs = ", ".join(f'"=&r"(r[{i}])' for i in range(64))
    print(f"""// two runs of 32 columns (early-clobber outputs: the second address is read after the first load has begun to write)
__device__ __forceinline__ void tmem_ld_2x32_wait(uint32_t first, uint32_t second, uint32_t (&r)[64]) {{
  asm volatile(
    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {{{regs(32, 0)}}}, [%64];\\n\\t"
    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {{{regs(32, 32)}}}, [%65];\\n\\t"
    "tcgen05.wait::ld.sync.aligned;\\n"
    : {outs}
    : "r"(first), "r"(second) : "memory");
}}
""")

def emit_ld_split(n):
    outs = ", ".join(f'"=r"(r[{i}])' for i in range(n))
    inouts = ", ".join(f'"+r"(r[{i}])' for i in range(n))
    print(f"""// a load without its wait, and the wait for it: the registers may not be touched in between
__device__ __forceinline__ void tmem_ld_x{n}(uint32_t taddr, uint32_t (&r)[{n}]) {{
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x{n}.b32 {{{regs(n, 0)}}}, [%{n}];"
    : {outs}
    : "r"(taddr) : "memory");
}}
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[{n}]) {{
  asm volatile("tcgen05.wait::ld.sync.aligned;" : {inouts} :: "memory");
}}
""")

def emit_st(n):
    ins = ", ".join(f'"r"(r[{i}])' for i in range(n))
    print(f"""__device__ __forceinline__ void tmem_st_x{n}(uint32_t taddr, const uint32_t (&r)[{n}]) {{
  asm volatile(
    "tcgen05.st.sync.aligned.32x32b.x{n}.b32 [%0], {{{regs(n, 1)}}};\\n"
    :: "r"(taddr), {ins} : "memory");
}}
""")

print("// Generated by gen_tmem_ops.py -- do not edit by hand.")
print("#pragma once")
print("#include <stdint.h>")
print("namespace ditto_b200 {")
for n in (8, 16, 32, 64, 128):
    emit_ld(n)
emit_ld_2x32()
emit_ld_split(32)
for n in (8, 16, 32, 64):
    emit_st(n)
print("}  // namespace ditto_b200")
