// What the kernels share that multiply float32 operands on the tensor cores: every float in three bfloat16 terms, terms in tensor
// memory (operand A) or shared memory (operand B), sums read back piece by piece.
#pragma once
#include "tc_common.cuh"

namespace plm_split {
using namespace plm_tc;

// A test build only (-DPLM_TEST_GIVE_UP, never the library that serves): while the switch is 1, the loader announces 64 bytes
// more for every stage than it loads, so that every wait runs out; while it is 2, one of the warps that add sums up acts as if
// its wait for the CTA's sixth stage had run out.  The kernel must record it, let what it has in flight land, free its tensor
// memory and return.
#ifdef PLM_TEST_GIVE_UP
__device__ int give_up_switch = 0;
#define PLM_STALL_BYTES (plm_split::give_up_switch == 1 ? 64u : 0u)
#define PLM_GIVES_UP(warp, stage) (plm_split::give_up_switch == 2 && (warp) == 3 && (stage) == 5)
#else
#define PLM_STALL_BYTES 0u
#define PLM_GIVES_UP(warp, stage) false
#endif

template <int NC> __device__ __forceinline__ void tmem_load(uint32_t addr, uint32_t (&r)[NC]) {
    static_assert(NC == 8 || NC == 16 || NC == 32, "columns");
    if constexpr (NC == 32) tc_ld32(addr, r);
    if constexpr (NC == 16)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                     "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(addr) : "memory");
    if constexpr (NC == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 "
                     "{%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(addr) : "memory");
}
// (the registers count as written by the wait, so that nothing made of them moves above it)
template <int NC> __device__ __forceinline__ void tmem_wait(uint32_t (&r)[NC]) {
    tc_wait_ld();
#pragma unroll
    for (int j = 0; j < NC; ++j) asm volatile("" : "+r"(r[j]));
}
__device__ __forceinline__ void tmem_store8(uint32_t addr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, uint32_t more) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a), "l"(b_desc), "r"(idesc), "r"(more) : "memory");
}

// What a float is multiplied by before it is split, and what a sum of products of two such is multiplied by.  bfloat16 has no bits
// below 2^-133, so the third term of a float below 2^-109 would be cut off, and more of it the smaller it is; 2^24 times as
// large all 24 bits of every float stand at 2^-125 and above, subnormal ones included.  What that sends beyond the largest
// float (operands from 2^104 on, sums from 2^80 on) becomes no number and is taken again with the other results of that kind.
constexpr float TERM_SCALE = 0x1p24f, SUM_SCALE = 0x1p-48f;

// two floats as pairs of bf16 terms; a and b become the remainders
__device__ __forceinline__ uint32_t next_terms(float& a, float& b) {
    const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
    const uint32_t w = *reinterpret_cast<const uint32_t*>(&t);
    a -= __uint_as_float(w << 16);
    b -= __uint_as_float(w & 0xffff0000u);
    return w;
}

}  // namespace plm_split

#ifdef PLM_TEST_GIVE_UP
extern "C" int plm_test_give_up(int how, cudaStream_t stream) {
    return plm_status_of(cudaMemcpyToSymbolAsync(plm_split::give_up_switch, &how, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
}
#endif
