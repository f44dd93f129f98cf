// C[M,N] = A[M,K] * W[N,K]^T in float32 on the tensor cores.  Sums of terms of both signs are as exact as float32 ones on the CUDA
// cores (gemm_simt.cu), sums of terms of one sign less so, see below.
//
// Every float (times 2^24, see TERM_SCALE) is the sum of three bfloat16 terms, exactly: h = bf16(x), m = bf16(x - h), l = x - h - m
// (24 bits of mantissa in three times 8, each remainder exact in fp32; a known way to split, as in S. Markidis et al., "NVIDIA
// Tensor Core Programmability, Performance & Precision", 2018).  A product of two terms has 16 bits and is exact in the tensor cores, so six
// products (hh, hm, mh, hl, lh, mm) leave out less than 2^-25 of a term: what remains is the rounding of the accumulator.
// Each STAGE of 32 terms of K is accumulated from zero, the small products first: a piece.  SETTLE pieces are added up in fp32, and
// their sum joins the two floats (head and rest) that hold the sum so far.
//
// The order of a result's sums is fixed by K alone: pieces of 32 terms in ascending order make a segment of SEGMENT
// terms, the segments' sums are added as doubles in ascending order, and the sum is rounded once.  So a row's result does not depend
// on how many rows stand beside it, though tiles have 16 to 96 rows of A and the segments of a tile may be dealt out to the
// CTAs of a cluster.
//
// What is not finite: an infinity's remainder is no number, so a result that is not finite (also after an overflow, which
// operands from 2^104 and sums from 2^80 on meet) is
// taken again from the rows themselves, by fused multiply-adds as gemm_simt.cu does.
//
// The error against 64 bits, in 2^-24 of the result (2-norm; K of 128 to 14,336), here and on the CUDA cores: rows of normal numbers
// times normal weights 1.18 to 1.22 and 1.31, rows silu(x) y of a gated feed-forward 1.26 to 1.28 and 1.28 to 1.31, both of a wide range
// (x^5, signed) 1.40 to 1.43 and 1.23 to 1.42.  An MMA cuts its addends off a few bits below the largest and truncates its
// sum, so terms of one sign come out low by 0.86: positive normal or uniform numbers 0.97 to 1.10 and 0.46 to 0.59; positive ones
// over several decades (e^(2x)), where one term of 16 outweighs the others, 2.5 to 5.5 and 0.6 to 1.5.  A model's weights have both signs.
// The longer the sums in fp32, the larger the error: pieces of 64 terms in one accumulator 5.3; of normal numbers and of silu(x) y SETTLE = 1
// 1.11 and 1.18, 2 1.17 and 1.24, 4 1.27 and 1.33, at 328, 250 and 226 us for 462 x 16,384 x 2,048 and 236 with 3.  A double's addition
// a piece: 1.05, but slow here (2,000 cycles a stage for 128 x 128 results).
// The CUDA cores against this: 462 rows x 16,384 x 2,048 893 and 236 us (131 TFLOP/s of float32 products); x 2,048 x 8,192 662 and 137;
// 24 rows x 3,072 x 2,048 42.7 and 17.3; 8 rows x 2,048 x 8,192 71 and 33.
// Bound by the chain of hand-overs between the warps and by their instructions (issue slots 62 to 69 % taken, the tensor pipe busy for
// 33 to 35 % of the time; an MMA takes 106 cycles at 96 columns, 79 at 64, 58 at 16, W's terms out of tensor memory among them).  Everything done by
// the same eight warps, with W's terms in shared memory too: 490 us for 462 x 2,048 x 8,192; splitting and adding apart 275;
// W's terms in tensor memory 237; two issuing warps behind elect.sync 190; four splitting warps a stage in turns 171
// (all of these with SETTLE = 4).
#include "split_common.cuh"

using namespace plm_tc;
using namespace plm_split;

namespace {

// Warps: eight add up pieces, two times four split every other stage each, one loads, two issue the MMAs (of every other
// stage), one fills the last group of four.  Registers are dealt out again at the start.
constexpr int FOLDERS = 8, GROUPS = 2, LOADER = FOLDERS + 4 * GROUPS, ISSUER = LOADER + 1, THREADS = 32 * (LOADER + 4);
constexpr int LAUNCH_REGS = 96, FOLD_REGS = 144, SPLIT_REGS = 80, REST_REGS = 32;
static_assert(32 * (FOLDERS * FOLD_REGS + 4 * GROUPS * SPLIT_REGS + 4 * REST_REGS) <= THREADS * LAUNCH_REGS && THREADS * LAUNCH_REGS <= 65536, "registers");
constexpr int SETTLE = 3;                                      // pieces that are summed in fp32 before their sum joins the head
constexpr int STAGE = 32, SEGMENT = 1024, SEGMENT_STAGES = SEGMENT / STAGE;    // a stage is a piece of 32 terms of K
constexpr int ROWS = 128;                                      // rows of W a tile (the MMA's M)

template <int NB> struct Tile {                                // NB rows of A a tile
    static constexpr int RAW = (ROWS + NB) * STAGE * 4;        // a stage as it comes from memory
    // W's terms go to tensor memory (a lane a row, two values a column), A's to shared memory: rows of 64 bytes with the
    // 64-byte swizzle.
    static constexpr int TERM_A = NB * STAGE * 2, TERMS = 3 * TERM_A;
    static constexpr int SENT = ROWS * NB * 8;                 // what the CTAs of a cluster send one another
    // tensor memory: two accumulators, the segments' sums (a double: two columns), two stages of W's terms
    static constexpr int SUMS = 2 * NB, TERMS_W = 4 * NB, COLUMNS = TERMS_W + 2 * 3 * STAGE / 2;
    static constexpr int TMEM = COLUMNS <= 128 ? 128 : COLUMNS <= 256 ? 256 : 512;
    __host__ __device__ static constexpr int ring(int cs) { return cs > 1 ? 4 : 6; }
    __host__ __device__ static constexpr int smem(int cs) { return ring(cs) * RAW + 2 * TERMS + (cs > 1 ? SENT : 0) + 1024; }
};

// Descriptor of a K-major bf16 tile with rows of 64 bytes and the 64-byte swizzle: eight rows are 512 bytes, layout type 4.
__device__ __forceinline__ uint64_t desc_sw64(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}

// Two floats at a time, each rounded as a sum of its own.
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(0xbf800000bf800000ull), "l"(a));
    return r;
}
// head + rest as the rounded sum and what it left out (Knuth's two-sum)
__device__ __forceinline__ void settle(uint64_t& head, uint64_t& rest) {
    const uint64_t t = add2(head, rest), b = sub2(t, head);
    rest = add2(sub2(head, sub2(t, b)), sub2(rest, b));
    head = t;
}

// The result of one row of A and one of W as gemm_simt.cu takes it.
__device__ __noinline__ float dot_again(const float* a, const float* w, int K) {
    double wide = 0.0;
    for (int k0 = 0; k0 < K; k0 += 16) {
        float acc = 0.f;
        for (int k = k0; k < K && k < k0 + 16; ++k) acc = fmaf(a[k], w[k], acc);
        wide += (double)acc;
    }
    return (float)wide;
}

struct F32Args {
    const float *A, *W;
    float* C;
    int M, N, K, row_tiles;
    long lda, ldw, ldc;
    int* status;
};

// A stage's way: copied in as it is (a ring of R), split by four warps (W's terms to tensor memory, A's to shared memory, two
// stages' worth), 12 MMAs into one of two accumulators, added up by eight warps.  terms_full stands for both "the terms are there"
// and "the accumulator is read", so that the issuing warp waits once a stage: a wait that is already over costs some 200 cycles.
// A tile of 128 rows of W x NB rows of A; the CS CTAs of a cluster take its segments in turn and each ends with every CS-th
// column of the tile.
template <int NB, int CS>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const F32Args g) {
    using T = Tile<NB>;
    constexpr int R = T::ring(CS), COLS = NB / 2;                  // COLS: columns a thread adds up
    constexpr uint32_t IDESC = instr_desc_bf16(NB);
    // a splitting warp that waits for a stage has been through the one before it in the same place of the ring
    static_assert(R % GROUPS == 0, "a phase could be taken for the one after the next");
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t bars[2 * R + 4];
    __shared__ uint32_t tmem_at;
    unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    unsigned char* terms = smem + R * T::RAW;
    double* sent = reinterpret_cast<double*>(terms + 2 * T::TERMS);
    const uint32_t bar0 = smem_u32(bars);
    auto raw_full = [&](int b) { return bar0 + 8 * b; };
    auto raw_empty = [&](int b) { return bar0 + 8 * (R + b); };
    auto terms_full = [&](int b) { return bar0 + 8 * (2 * R + b); };
    auto mma_done = [&](int b) { return bar0 + 8 * (2 * R + 2 + b); };
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int rank = CS > 1 ? (int)cluster_rank() : 0;
    const int tile = blockIdx.x / CS;
    const int m0 = (tile % g.row_tiles) * NB, n0 = (tile / g.row_tiles) * ROWS;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_at)), "r"(T::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int b = 0; b < R; ++b) {
            mbar_init(raw_full(b), 1);
            mbar_init(raw_empty(b), 4);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(terms_full(b), 4 + FOLDERS);    // the terms are there and the accumulator is read
            mbar_init(mma_done(b), 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if constexpr (CS > 1) cluster_sync_all();                  // every CTA has begun before one writes to its memory
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_at, 0);

    // A cluster's CTAs take one segment each a round; a CTA alone has all stages in one round.
    const int n_stages_all = (g.K + STAGE - 1) / STAGE, n_segments = (n_stages_all + SEGMENT_STAGES - 1) / SEGMENT_STAGES;
    const int n_rounds = CS > 1 ? (n_segments + CS - 1) / CS : 1;
    auto first_of = [&](int round) { return CS > 1 ? (round * CS + rank) * SEGMENT_STAGES : 0; };
    auto stages_of = [&](int round) { return CS > 1 ? max(0, min(SEGMENT_STAGES, n_stages_all - first_of(round))) : n_stages_all; };
    bool ok = true;
    int done = 0;                                              // stages of the rounds before
    // (a warp whose wait runs out arrives nowhere any more, so that those behind it give up as well, and each meets its cluster's
    // barriers all the same)
    if (warp >= LOADER) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REST_REGS));
        int asked = 0;                                         // stages that the loader has asked for
        for (int round = 0; round < n_rounds; ++round) {
            const int first = first_of(round), n_stages = stages_of(round);
            if (warp == LOADER && lane == 0) {
                for (int s = 0; s < n_stages && ok; ++s, ++asked) {
                    const int at = asked, b = at % R;
                    if (at >= R) ok = mbar_wait(raw_empty(b), ((at - R) / R) & 1, g.status, 60);
                    if (!ok) break;
                    mbar_expect_tx(raw_full(b), T::RAW + PLM_STALL_BYTES);
                    tma_load_2d(smem_u32(smem + b * T::RAW), &map_w, raw_full(b), (first + s) * STAGE, n0);
                    tma_load_2d(smem_u32(smem + b * T::RAW + ROWS * STAGE * 4), &map_a, raw_full(b), (first + s) * STAGE, m0);
                }
            } else if (warp == ISSUER || warp == ISSUER + 1) {
                // two warps, so that one's waits pass while the other's MMAs run; the smallest products first
                const int b = warp - ISSUER;
                const uint32_t w = tmem + T::TERMS_W + b * 48, d = tmem + b * NB;
                const uint64_t a = desc_sw64(smem_u32(terms + b * T::TERMS));
                for (int s = (done ^ b) & 1; s < n_stages && ok; s += 2) {
                    ok = mbar_wait_warp(terms_full(b), ((done + s) >> 1) & 1, g.status, 61);
                    if (!ok) break;
                    tc_fence_after();
                    constexpr int TW[6] = {1, 2, 0, 1, 0, 0}, TA[6] = {1, 0, 2, 0, 1, 0};
                    if (elect_one()) {
#pragma unroll
                        for (int p = 0; p < 6; ++p)
#pragma unroll
                            for (int k = 0; k < STAGE / UMMA_K; ++k)
                                mma_ts(d, w + TW[p] * 16 + k * 8, a + (TA[p] * T::TERM_A + k * 32) / 16, IDESC, p + k > 0);
                        tc_commit(mma_done(b));
                    }
                    __syncwarp();
                }
            }
            __syncwarp();
            done += n_stages;
            if constexpr (CS > 1) {
                if (round > 0) cluster_sync_all();
                cluster_sync_all();
            }
        }
        if (warp == LOADER && lane == 0)                       // no copy may be under way when the CTA ends, whoever gave up
            for (int i = max(0, asked - R); i < asked; ++i) mbar_wait(raw_full(i % R), (i / R) & 1, nullptr, 0);
        __syncwarp();
    } else if (warp >= FOLDERS) {
        // split: of W a lane a row, of A eight terms of a row at a time
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(SPLIT_REGS));
        const int group = (warp - FOLDERS) / 4, member = warp % 4, a_row = lane % 8, q = lane / 8;
        const uint32_t w_to = tmem + ((uint32_t)(member * 32) << 16) + T::TERMS_W;
        for (int round = 0; round < n_rounds; ++round) {
            const int n_stages = stages_of(round);
            for (int s = (group + GROUPS - done % GROUPS) % GROUPS; s < n_stages && ok; s += GROUPS) {
                const int at = done + s, b = at % R;
                ok = mbar_wait_warp(raw_full(b), (at / R) & 1, g.status, 62);
                if (!ok) break;
                const unsigned char* raw = smem + b * T::RAW;
                uint32_t w[2][3][8];                           // (before the MMAs that read the buffers last are waited for)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float x[16];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        *reinterpret_cast<float4*>(x + 4 * i) = *reinterpret_cast<const float4*>(raw + (member * 32 + lane) * 128 + ((4 * h + i) ^ (lane % 8)) * 16);
#pragma unroll
                    for (int i = 0; i < 16; ++i) x[i] *= TERM_SCALE;
#pragma unroll
                    for (int t = 0; t < 3; ++t)
#pragma unroll
                        for (int i = 0; i < 8; ++i) w[h][t][i] = next_terms(x[2 * i], x[2 * i + 1]);
                }
                if (at >= 2) ok = mbar_wait_warp(mma_done(at & 1), ((at - 2) >> 1) & 1, g.status, 62);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int t = 0; t < 3; ++t) tmem_store8(w_to + (at & 1) * 48 + t * 16 + h * 8, w[h][t]);
                raw += ROWS * STAGE * 4 + a_row * 128;
                unsigned char* to = terms + (at & 1) * T::TERMS + a_row * 64 + (q ^ (a_row >> 1)) * 16;
#pragma unroll
                for (int block = member; block < NB / 8; block += 4) {             // of eight rows
                    float x[8];
                    *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(raw + block * 1024 + ((2 * q) ^ a_row) * 16);
                    *reinterpret_cast<float4*>(x + 4) = *reinterpret_cast<const float4*>(raw + block * 1024 + ((2 * q + 1) ^ a_row) * 16);
#pragma unroll
                    for (int i = 0; i < 8; ++i) x[i] *= TERM_SCALE;
#pragma unroll
                    for (int t = 0; t < 3; ++t) {
                        uint4 v;
                        v.x = next_terms(x[0], x[1]);
                        v.y = next_terms(x[2], x[3]);
                        v.z = next_terms(x[4], x[5]);
                        v.w = next_terms(x[6], x[7]);
                        *reinterpret_cast<uint4*>(to + t * T::TERM_A + block * 512) = v;
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(terms_full(at & 1));
                    mbar_arrive(raw_empty(b));
                }
            }
            __syncwarp();
            done += n_stages;
            if constexpr (CS > 1) {
                if (round > 0) cluster_sync_all();
                cluster_sync_all();
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FOLD_REGS));
        const uint32_t lanes = tmem + ((uint32_t)(warp % 4 * 32) << 16), half = (warp / 4) * COLS;
        uint64_t head[COLS / 2], rest[COLS / 2];               // two columns each: a column's sum is head + rest
        double total[CS > 1 ? COLS / CS : 1];
#pragma unroll
        for (int j = 0; j < COLS / 2; ++j) head[j] = rest[j] = 0;
#pragma unroll
        for (int j = 0; j < (CS > 1 ? COLS / CS : 1); ++j) total[j] = 0.0;
        auto sum_of = [&](int j) {
            const uint32_t h = (uint32_t)(head[j / 2] >> (32 * (j & 1))), r = (uint32_t)(rest[j / 2] >> (32 * (j & 1)));
            return (double)__uint_as_float(h) + (double)__uint_as_float(r);
        };
        if (lane == 0) {                                       // both accumulators are free
            mbar_arrive(terms_full(0));
            mbar_arrive(terms_full(1));
        }
        __syncwarp();
        for (int round = 0; round < n_rounds; ++round) {
            const int n_stages = stages_of(round);
            for (int s = 0; s < n_stages && ok; ++s) {
                const int at = done + s, b = at & 1;
                ok = mbar_wait_warp(mma_done(b), (at >> 1) & 1, g.status, 63);
                if (PLM_GIVES_UP(warp, at)) {
                    atomicCAS(g.status, 0, 63);
                    ok = false;
                }
                if (!ok) break;
                tc_fence_after();
                auto take = [&](auto& r, int c) {
                    constexpr int n = sizeof(r) / 4;
                    tmem_load<n>(lanes + b * NB + half + c, r);
                    tmem_wait<n>(r);
                    if (c + n == COLS) {                       // the accumulator is read
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(terms_full(b));
                    }
#pragma unroll
                    for (int j = 0; j < n; j += 2) rest[(c + j) / 2] = add2(rest[(c + j) / 2], (uint64_t)r[j + 1] << 32 | r[j]);
                };
#pragma unroll
                for (int c = 0; c + 32 <= COLS; c += 32) {
                    uint32_t r[32];
                    take(r, c);
                }
                if constexpr (COLS % 32 > 0) {
                    uint32_t r[COLS % 32];
                    take(r, COLS / 32 * 32);
                }
                const int in_segment = s % SEGMENT_STAGES + 1;
                if (in_segment % SETTLE == 0)
#pragma unroll
                    for (int j = 0; j < COLS / 2; ++j) settle(head[j], rest[j]);
                if (CS == 1 && in_segment == SEGMENT_STAGES && s + 1 < n_stages) {
                    // a segment ends: its sums join those in front of it, in tensor memory (a double: two columns)
                    const uint32_t sums = lanes + T::SUMS + 2 * half;
#pragma unroll
                    for (int c = 0; c < COLS; c += 4) {
                        uint32_t r[8];
                        const bool before = s >= SEGMENT_STAGES;
                        if (before) {
                            tmem_load<8>(sums + 2 * c, r);
                            tmem_wait<8>(r);
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            double v = sum_of(c + j);
                            if (before) v = __hiloint2double((int)r[2 * j + 1], (int)r[2 * j]) + v;
                            r[2 * j] = (uint32_t)__double2loint(v);
                            r[2 * j + 1] = (uint32_t)__double2hiint(v);
                        }
                        tmem_store8(sums + 2 * c, r);
                        head[c / 2] = head[c / 2 + 1] = rest[c / 2] = rest[c / 2 + 1] = 0;
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                }
            }
            done += n_stages;
            if constexpr (CS > 1) {
                if (round > 0) cluster_sync_all();             // what the last round sent is added up
#pragma unroll
                for (int j = 0; j < COLS; ++j) {
                    const uint32_t to = cluster_map(&sent[(rank * (COLS / CS) + j / CS) * (32 * FOLDERS) + tid], j % CS);
                    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(to), "d"(sum_of(j)) : "memory");
                }
#pragma unroll
                for (int j = 0; j < COLS / 2; ++j) head[j] = rest[j] = 0;
                cluster_sync_all();
                for (int r = 0; r < CS && round * CS + r < n_segments; ++r)
#pragma unroll
                    for (int j = 0; j < COLS / CS; ++j) total[j] += sent[(r * (COLS / CS) + j) * (32 * FOLDERS) + tid];
            }
        }
        // (the stores first and what is not finite behind them: a look at each result on its way out takes some 200 cycles)
        const int n = n0 + warp % 4 * 32 + lane;
        const uint32_t sums = lanes + T::SUMS + 2 * half;
        constexpr int STEP = CS > 1 ? CS : 1;                  // from one of this thread's columns to the next
        const int first = m0 + half + (CS > 1 ? rank : 0), count = ok ? min(COLS / STEP, (g.M - first + STEP - 1) / STEP) : 0;
        float* to = g.C + (size_t)first * g.ldc + n;
        const size_t ld = (size_t)STEP * g.ldc;
        bool finite = true;
#pragma unroll
        for (int c = 0; c < COLS / STEP; c += CS > 1 ? 1 : 4) {
            uint32_t r[8];
            if (CS == 1 && n_segments > 1) {
                tmem_load<8>(sums + 2 * c, r);
                tmem_wait<8>(r);
            }
#pragma unroll
            for (int j = 0; j < (CS > 1 ? 1 : 4); ++j) {
                double wide = CS > 1 ? total[CS > 1 ? c : 0] : sum_of(c + j);
                if (CS == 1 && n_segments > 1) wide = __hiloint2double((int)r[2 * j + 1], (int)r[2 * j]) + wide;
                const float v = (float)wide * SUM_SCALE;
                if (n < g.N && c + j < count) {
                    finite = finite && fabsf(v) <= 3.402823466e38f;
                    to[(c + j) * ld] = v;
                }
            }
        }
        if (!finite)
#pragma unroll 1
            for (int j = 0; j < count; ++j)
                if (!(fabsf(to[j * ld]) <= 3.402823466e38f))
                    to[j * ld] = dot_again(g.A + (size_t)(first + j * STEP) * g.lda, g.W + (size_t)n * g.ldw, g.K);
        __syncwarp();
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::TMEM) : "memory");
}

// A [rows, K] float32 matrix of leading dimension ld, boxes of box_rows x 32; kept by what they describe, as make_map's.
int make_map_f32(CUtensorMap* map, const void* ptr, long rows, long K, long ld, int box_rows) {
    struct Entry { const void* ptr; long rows, K, ld; int box_rows; bool used; CUtensorMap map; };
    constexpr int SLOTS = 256;
    static Entry table[SLOTS];
    static std::mutex lock;
    const size_t h = ((size_t)ptr >> 4) * 0x9E3779B97F4A7C15ull + (size_t)rows * 31 + (size_t)K * 131 + (size_t)box_rows;
    Entry& e = table[(h >> 20) % SLOTS];
    {
        std::lock_guard<std::mutex> g(lock);
        if (e.used && e.ptr == ptr && e.rows == rows && e.K == K && e.ld == ld && e.box_rows == box_rows) {
            *map = e.map;
            return PLM_OK;
        }
    }
    EncodeTiledFn fn = encode_fn();
    if (!fn) return PLM_ERR_UNSUPPORTED;
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
    cuuint32_t box[2] = {(cuuint32_t)STAGE, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    if (fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return PLM_ERR_ALIGN;
    std::lock_guard<std::mutex> g(lock);
    e.ptr = ptr; e.rows = rows; e.K = K; e.ld = ld; e.box_rows = box_rows; e.map = *map; e.used = true;
    return PLM_OK;
}

template <int NB, int CS>
int launch_f32_tc(F32Args g, cudaStream_t stream) {
    static std::atomic<unsigned long long> devices{0};
    constexpr int SMEM = Tile<NB>::smem(CS);
    static_assert(SMEM <= 232448 - 256 && Tile<NB>::TMEM <= 512, "an SM's memory");
    const cudaError_t configured = plm_allow_smem(gemm_f32_tc_kernel<NB, CS>, SMEM, devices);
    if (configured != cudaSuccess) return (int)configured;
    g.row_tiles = (g.M + NB - 1) / NB;
    const long tiles = (long)g.row_tiles * ((g.N + ROWS - 1) / ROWS);
    if (tiles * CS > 0x7fffffffL) return PLM_ERR_SHAPE;
    CUtensorMap map_w, map_a;
    int r = make_map_f32(&map_w, g.W, g.N, g.K, g.ldw, ROWS);
    if (r == PLM_OK) r = make_map_f32(&map_a, g.A, g.M, g.K, g.lda, NB);
    if (r != PLM_OK) return r;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * CS));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = CS > 1 ? 1 : 0;
    return plm_status_of(cudaLaunchKernelEx(&cfg, gemm_f32_tc_kernel<NB, CS>, map_w, map_a, g));
}

template <int NB>
int launch_rows(int cluster, const F32Args& g, cudaStream_t stream) {
    if (cluster == 8) return launch_f32_tc<NB, 8>(g, stream);
    if (cluster == 4) return launch_f32_tc<NB, 4>(g, stream);
    if (cluster == 2) return launch_f32_tc<NB, 2>(g, stream);
    return launch_f32_tc<NB, 1>(g, stream);
}

// The form whose waves of CTAs take the least time, as rows of A a tile + 1000 * CTAs a tile.  Cycles of a stage and of what a
// CTA does beside its stages (its start, the sums' exchange, the stores) are measured; the model is within a tenth of the
// times from 1 to 1,300 rows (2,048 to 32,000 columns, K of 2,048 and 8,192).
int f32_tc_form(int M, int N, int K) {
    constexpr int NBS[4] = {16, 32, 64, 96}, CYCLES[4] = {740, 780, 1000, 1250};
    const int stages = (K + STAGE - 1) / STAGE, segments = (stages + SEGMENT_STAGES - 1) / SEGMENT_STAGES;
    int best = 0;
    double best_cycles = 0;
    for (int i = 0; i < 4; ++i)
        for (int cs = 1; cs <= (NBS[i] == 96 ? 1 : 8); cs *= 2) {
            if (cs > 1 && cs >= 2 * segments) break;           // half of the cluster would stand idle
            const long ctas = (long)((M + NBS[i] - 1) / NBS[i]) * ((N + ROWS - 1) / ROWS) * cs;
            const long waves = (ctas + PLM_SM_COUNT - 1) / PLM_SM_COUNT;
            const int rounds = (segments + cs - 1) / cs;
            const double cycles = waves * ((cs > 1 ? (double)rounds * (stages < SEGMENT_STAGES ? stages : SEGMENT_STAGES) : stages) * CYCLES[i] +
                                           (cs > 1 ? 14500.0 * rounds : 12500.0));
            if (!best || cycles < best_cycles) {
                best = NBS[i] + 1000 * cs;
                best_cycles = cycles;
            }
        }
    return best;
}

}  // namespace

// All three float32; K, lda and ldw multiples of 4, A and W on 16-byte boundaries.  form: 0 chooses, else one of
// plm_gemm_f32_tc_form's.
extern "C" int plm_gemm_f32_tc(const void* A, const void* W, void* C, int M, int N, int K, long lda, long ldw, long ldc, int form,
                               int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return PLM_OK;
    if (K <= 0 || lda < K || ldw < K || ldc < N || M > 64L * 65535) return PLM_ERR_SHAPE;   // (rows: as gemm_simt.cu)
    if (K % 4 || lda % 4 || ldw % 4 || (((uintptr_t)A | (uintptr_t)W) & 15)) return PLM_ERR_ALIGN;
    const F32Args g = {(const float*)A, (const float*)W, (float*)C, M, N, K, 0, lda, ldw, ldc, status};
    if (!form) form = f32_tc_form(M, N, K);
    const int rows = form % 1000, cluster = form / 1000;
    if (cluster != 1 && cluster != 2 && cluster != 4 && cluster != 8) return PLM_ERR_UNSUPPORTED;
    if (rows == 16) return launch_rows<16>(cluster, g, stream);
    if (rows == 32) return launch_rows<32>(cluster, g, stream);
    if (rows == 64) return launch_rows<64>(cluster, g, stream);
    return rows == 96 && cluster == 1 ? launch_f32_tc<96, 1>(g, stream) : PLM_ERR_UNSUPPORTED;
}

extern "C" int plm_gemm_f32_tc_form(int M, int N, int K) { return f32_tc_form(M, N, K); }
