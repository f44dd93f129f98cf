// Linear attention with one constant decay a head over rotated queries and keys, for prompts, in bfloat16 on tcgen05: the
// recurrence of decay_chunk.cu taken 128 tokens at a time.  With S the state before a chunk of n tokens,
//   o_t = d^(t+1) S^T q_t + sum_{s <= t} d^(t-s) (q_t . k_s) v_s
//   S  <- d^n S + sum_s k_s (d^(n-1-s) v_s)^T
// in three kernels: what every chunk adds to the state, all side by side (decay_add_kernel); the state at every chunk's start,
// a multiply and an add per value and chunk (decay_states_kernel); the outputs, all chunks side by side (decay_out_kernel).
//
// Precision is decay_chunk.cu's: v as it is, everything else (rotated queries and keys, decayed keys, the chunk's weights, the
// state where it is read) in two bf16 terms, x = hi + lo; a product of two such is hi hi + hi lo + lo hi.  The state itself is
// fp32.
//
// Why beside decay_chunk.cu: `mma.sync` runs at an eighth of tcgen05's rate here (some 16 cycles an m16n8k16 and scheduler), and
// that kernel spends its time on it.  16 heads of 128 x 256, us there / here: one sequence of 2,048 tokens 107 / 65, of 256 35 / 24, of 129
// 25 / 22; 8 heads of 64 x 128, 300 tokens and eight of 16 30 / 20.  Many short sequences leave the chunks half empty and run there
// (which step runs where: ops/recurrent.py, decay_in_128).  Of the 65 the outputs are 41 (a CTA's phases follow one another: loads and
// rotation, products, results), the chunks' sums 19, the states 10.  Errors against 64 bits, there / here (the 16 bits of what is kept in
// two terms): 5.9e-6 / 5.1e-6 of 2,048 tokens' outputs, 4.1e-6 / 2.5e-6 of the state.
//
// What is not finite in a token's v goes in as zero and makes the outputs of its column no numbers from that token on, so that
// the zero weights of earlier tokens make none of it; in the state it stays as it is.
#include "mma_common.cuh"
#include "split_common.cuh"

namespace {

constexpr int C = 128, PT = 128;                       // tokens of a chunk; value columns of a unit
constexpr uint32_t ROWS_64 = C * 128;                  // bytes of 128 rows of 64 bf16 values, 128-byte swizzle

struct DecayArgs {
    const bf16 *q, *k, *v;
    long ldq, ldk, ldv;
    const float* powers;                               // [H][65]: d^0 .. d^64
    float* state;
    long state_stride;
    float* y;
    long ldy;
    const int *seq_start, *seq_slot;
    int n_seqs, H, N, P;
    const float *cos_t, *sin_t;
    const int* tok_pos;
    int half;
    float k_scale;
    float* ws;                                         // [slot][H][N][P]: what a chunk adds
    bf16* states;                                      // [slot][H][2][N][P]: the state at its start in two terms
    int* status;
    int tiles, per;                                    // value tiles of a head; how many of them a CTA takes
    // a chunk's place: a sequence's lie one behind the other
    __device__ long slot(int s0, int b, int c) const { return s0 / C + b + c; }
};

// A block's chunk, head and value tiles.  Blocks stand for the chunks' places and not for every sequence's chunks up to the longest
// one's, so at most one place a sequence is empty: a block finds its chunk's sequence by a warp's search over the places where
// sequences begin.  (A block for every sequence and chunk of the longest: 2,000 tokens beside 63 of 1, 16 heads of 128 x 256, 547 us for 334;
// 700 beside 20 of 60 with a captured step's bounds 241 for 140.)
struct Where { int b, h, c, p0, t0, n; };
__device__ __forceinline__ Where where_of(const DecayArgs& a) {
    Where w;
    unsigned u = blockIdx.x;
    const unsigned parts = (unsigned)((a.tiles + a.per - 1) / a.per);
    w.p0 = (int)(u % parts) * a.per * PT, u /= parts;
    w.h = (int)(u % (unsigned)a.H);
    const int place = (int)(u / (unsigned)a.H), lane = threadIdx.x & 31;
    int s0, s1;
    if (a.n_seqs < 32) {                               // all of them in one load
        const int start = a.seq_start[min(lane, a.n_seqs)];
        const bool begun = lane < a.n_seqs && (int)a.slot(start, lane, 0) <= place;
        w.b = max(__popc(__ballot_sync(0xffffffffu, begun)) - 1, 0);             // (places ascend)
        s0 = __shfl_sync(0xffffffffu, start, w.b), s1 = __shfl_sync(0xffffffffu, start, w.b + 1);
    } else {
        int hi = a.n_seqs;                             // the sequence is one from w.b on and before this
        w.b = 0;
        while (hi - w.b > 1) {
            const int step = (hi - w.b + 31) / 32, b = w.b + lane * step;
            const bool begun = b < hi && (int)a.slot(a.seq_start[b], b, 0) <= place;
            w.b += max(__popc(__ballot_sync(0xffffffffu, begun)) - 1, 0) * step;
            hi = min(hi, w.b + step);
        }
        s0 = a.seq_start[w.b], s1 = a.seq_start[w.b + 1];
    }
    w.c = place - (int)a.slot(s0, w.b, 0);
    w.t0 = s0 + w.c * C;
    w.n = w.c < 0 ? 0 : min(C, s1 - w.t0);
    return w;
}
// d^e for e of 0 .. 128 from the table of 65
__device__ __forceinline__ float power_of(const float* pw, int e) { return e <= 64 ? pw[e] : pw[64] * pw[e - 64]; }

// where column c of row r lies in blocks of 64 columns
__device__ __forceinline__ uint32_t place(int r, int c) { return (uint32_t)(c >> 6) * ROWS_64 + (uint32_t)r * 128 + ((((uint32_t)c >> 3) & 7) ^ ((uint32_t)r & 7)) * 16; }

// Eight pairs of a row turned by their angles and multiplied, as two terms each, to places cu and cv of row r.
__device__ __forceinline__ void turn_to(const uint4& u, const uint4& v, bool turn, const float4 (&cs)[4], float scale, uint8_t* hi, uint8_t* lo, int r, int cu, int cv) {
    const uint32_t *uw = reinterpret_cast<const uint32_t*>(&u), *vw = reinterpret_cast<const uint32_t*>(&v);
    const float *c = reinterpret_cast<const float*>(cs), *sn = c + 8;
    uint32_t uh[4], ul[4], vh[4], vl[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 x = bf16_pair(uw[i]), y = bf16_pair(vw[i]);
        float2 p = x, q = y;
        if (turn) {
            p = make_float2(rope_first(x.x, y.x, c[2 * i], sn[2 * i]), rope_first(x.y, y.y, c[2 * i + 1], sn[2 * i + 1]));
            q = make_float2(rope_second(x.x, y.x, c[2 * i], sn[2 * i]), rope_second(x.y, y.y, c[2 * i + 1], sn[2 * i + 1]));
        }
        split2(p.x * scale, p.y * scale, uh[i], ul[i]);
        split2(q.x * scale, q.y * scale, vh[i], vl[i]);
    }
    *reinterpret_cast<uint4*>(hi + place(r, cu)) = make_uint4(uh[0], uh[1], uh[2], uh[3]);
    *reinterpret_cast<uint4*>(lo + place(r, cu)) = make_uint4(ul[0], ul[1], ul[2], ul[3]);
    *reinterpret_cast<uint4*>(hi + place(r, cv)) = make_uint4(vh[0], vh[1], vh[2], vh[3]);
    *reinterpret_cast<uint4*>(lo + place(r, cv)) = make_uint4(vl[0], vl[1], vl[2], vl[3]);
}
__device__ __forceinline__ void angles(const DecayArgs& a, long pos, int g8, bool in, float4 (&cs)[4]) {
    if (in) {
        const float4 *cp = reinterpret_cast<const float4*>(a.cos_t + pos * a.half + g8), *sp = reinterpret_cast<const float4*>(a.sin_t + pos * a.half + g8);
        cs[0] = cp[0], cs[1] = cp[1], cs[2] = sp[0], cs[3] = sp[1];
    } else {
        cs[0] = cs[1] = cs[2] = cs[3] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
// whether one of eight bf16 values is not finite
__device__ __forceinline__ bool odd_one(uint32_t w) { return (w & 0x7f80u) == 0x7f80u || (w & 0x7f800000u) == 0x7f800000u; }

// K-major: rows of 64 values, 16 of them a step; MN-major: eight rows of K 1,024 bytes apart, blocks of 64 columns ROWS_64
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr, uint32_t block) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(block >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ void alloc_tmem(uint32_t slot, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void store16(uint32_t addr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                   "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}

// ---------------------------------------------------------------- what a chunk adds: sum_s k_s (d^(n-1-s) v_s)^T
// D[p][n]: v on the MMA's rows, the decayed keys its columns, both as they lie (rows of tokens, their columns contiguous).
constexpr int ADD_NT = 256;
template <int NP> constexpr size_t add_smem() { return 2 * (NP / 64) * ROWS_64 + 2 * ROWS_64 + 1024; }

template <int NP>
__global__ void __launch_bounds__(ADD_NT, 2) decay_add_kernel(const DecayArgs a) {
    constexpr int PG = NP / 16;                        // groups of eight pairs in a row
    // M = 128, N = NP, D fp32, A and B bf16, both with their columns contiguous
    constexpr uint32_t IDESC = plm_tc::instr_desc_bf16(NP) | (1u << 15) | (1u << 16);
    extern __shared__ uint8_t add_raw[];
    __shared__ uint64_t bar;
    __shared__ uint32_t slot;
    __shared__ float pw[65];
    uint8_t* smem = add_raw + ((1024 - (plm_tc::smem_u32(add_raw) & 1023)) & 1023);
    uint8_t *khi = smem, *klo = khi + NP / 64 * ROWS_64, *vs = klo + NP / 64 * ROWS_64;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    pdl_launch_dependents();
    if (warp == 0) alloc_tmem(plm_tc::smem_u32(&slot), NP);
    const uint32_t done = plm_tc::smem_u32(&bar);
    if (tid == 0) {
        plm_tc::mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_wait();
    const Where w = where_of(a);
    for (int i = tid; i < 65; i += ADD_NT) pw[i] = a.powers[w.h * 65 + i];
    plm_tc::tc_fence_before();
    __syncthreads();
    plm_tc::tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, slot, 0);
    if (w.n > 0) {
        const long pos0 = a.half > 0 ? a.tok_pos[w.t0] : 0;
        // (loads before stores: shared and global memory are one to the compiler)
        constexpr int BATCH = 2;
        static_assert(C * PG / ADD_NT % BATCH == 0, "groups");
        const int tiles = min(a.per, a.tiles - w.p0 / PT);
        auto load_v = [&](int it) {                    // eight values of a row of v a thread, straight to their places
#pragma unroll
            for (int i = 0; i < C * 16 / ADD_NT; ++i) {
                const int idx = tid + i * ADD_NT, r = idx / 16, c = idx % 16 * 8;
                const bool in = r < w.n;
                cp_async16(plm_tc::smem_u32(vs) + place(r, c), a.v + (long)(w.t0 + (in ? r : 0)) * a.ldv + (long)w.h * a.P + w.p0 + it * PT + c, in);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        load_v(0);
#pragma unroll
        for (int i0 = 0; i0 < C * PG / ADD_NT; i0 += BATCH) {
            float4 cs[BATCH][4];
            uint4 x[BATCH][2];
#pragma unroll
            for (int i = 0; i < BATCH; ++i) {
                const int idx = tid + (i0 + i) * ADD_NT, r = idx / PG, g = idx % PG;
                const bool turn = g * 8 < a.half, in = r < w.n;
                const int cu = turn ? g * 8 : 2 * a.half + (g - a.half / 8) * 16, cv = turn ? a.half + g * 8 : cu + 8;
                x[i][0] = x[i][1] = make_uint4(0, 0, 0, 0);
                if (in) {
                    const bf16* row = a.k + (long)(w.t0 + r) * a.ldk + (long)w.h * NP;
                    x[i][0] = *reinterpret_cast<const uint4*>(row + cu), x[i][1] = *reinterpret_cast<const uint4*>(row + cv);
                }
                angles(a, pos0 + r, g * 8, turn && in, cs[i]);
            }
#pragma unroll
            for (int i = 0; i < BATCH; ++i) {
                const int idx = tid + (i0 + i) * ADD_NT, r = idx / PG, g = idx % PG;
                const bool turn = g * 8 < a.half;
                const int cu = turn ? g * 8 : 2 * a.half + (g - a.half / 8) * 16, cv = turn ? a.half + g * 8 : cu + 8;
                const float decay = r < w.n ? power_of(pw, w.n - 1 - r) : 0.f;
                turn_to(x[i][0], x[i][1], turn, cs[i], a.k_scale * decay, khi, klo, r, cu, cv);
            }
        }
        const int c0 = warp / 4 * (NP / 2);
        float* to = a.ws + (a.slot(a.seq_start[w.b], w.b, w.c) * a.H + w.h) * (long)NP * a.P + (long)c0 * a.P + w.p0 + warp % 4 * 32 + lane;
        for (int it = 0; it < tiles; ++it, to += PT) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            plm_tc::tc_fence_before();
            __syncthreads();
            if (warp == 0) {
                plm_tc::tc_fence_after();
                if (plm_tc::elect_one()) {
                    const uint64_t va = desc_mn(plm_tc::smem_u32(vs), ROWS_64);
#pragma unroll
                    for (int term = 0; term < 2; ++term) {
                        const uint64_t kb = desc_mn(plm_tc::smem_u32(term ? khi : klo), ROWS_64);
#pragma unroll
                        for (int s = 0; s < C / 16; ++s) plm_tc::tc_mma_bf16(tmem, va + s * 2048 / 16, kb + s * 2048 / 16, IDESC, term + s > 0);
                    }
                    plm_tc::tc_commit(done);
                }
                __syncwarp();
            }
            plm_tc::mbar_wait_warp(done, it & 1, a.status, 48);
            plm_tc::tc_fence_after();
            if (it + 1 < tiles) load_v(it + 1);
#pragma unroll
            for (int c = 0; c < NP / 2; c += 32) {
                uint32_t r[32];
                plm_split::tmem_load<32>(tmem + ((uint32_t)(warp % 4 * 32) << 16) + c0 + c, r);
                plm_split::tmem_wait<32>(r);
#pragma unroll
                for (int j = 0; j < 32; ++j) to[(long)(c + j) * a.P] = __uint_as_float(r[j]);
            }
        }
    }
    plm_tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NP) : "memory");
}

// ---------------------------------------------------------------- the state at every chunk's start
// A thread four columns of one row.
constexpr int STATES_NT = 128;
__global__ void __launch_bounds__(STATES_NT) decay_states_kernel(const DecayArgs a) {
    constexpr int AHEAD = 8;
    pdl_launch_dependents();
    pdl_wait();
    const long idx = (long)blockIdx.x * STATES_NT + threadIdx.x, quads = (long)a.N * a.P / 4;
    const int b = blockIdx.y, h = (int)(idx / quads);
    const int s0 = a.seq_start[b], len = a.seq_start[b + 1] - s0, n_chunks = (len + C - 1) / C;
    if (h >= a.H || len <= 0) return;
    const long at = idx % quads * 4, step = (long)a.H * a.N * a.P;
    const float* pw = a.powers + h * 65;
    float* st = a.state + (long)a.seq_slot[b] * a.state_stride + (long)h * a.N * a.P + at;
    const float* w = a.ws + a.slot(s0, b, 0) * step + (long)h * a.N * a.P + at;
    bf16* terms = a.states + 2 * (a.slot(s0, b, 0) * step + (long)h * a.N * a.P) + at;
    float4 S = *reinterpret_cast<const float4*>(st);
    for (int c0 = 0; c0 < n_chunks; c0 += AHEAD) {
        float4 add[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < n_chunks) add[i] = *reinterpret_cast<const float4*>(w + (c0 + i) * step);
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < n_chunks) {
                uint32_t h0, l0, h1, l1;
                split2(S.x, S.y, h0, l0);
                split2(S.z, S.w, h1, l1);
                bf16* to = terms + 2 * (c0 + i) * step;
                *reinterpret_cast<uint2*>(to) = make_uint2(h0, h1);
                *reinterpret_cast<uint2*>(to + (long)a.N * a.P) = make_uint2(l0, l1);
                const int n = len - (c0 + i) * C;
                // (in two steps: the rounding of d^64 squared would be the same in every chunk)
                const float d = pw[min(n, 64)], e = pw[max(min(n, C) - 64, 0)];
                S = make_float4(fmaf(d, S.x * e, add[i].x), fmaf(d, S.y * e, add[i].y), fmaf(d, S.z * e, add[i].z), fmaf(d, S.w * e, add[i].w));
            }
    }
    *reinterpret_cast<float4*>(st) = S;
}

// ---------------------------------------------------------------- the outputs
// Tokens on the MMA's rows.  Sixteen warps bring in queries and keys, then (while those are multiplied) values and state, and
// make of the scores the weights d^(t-s) q.k, which go back to tensor memory in two terms as the third product's operand A; a
// seventeenth issues, so that nobody waits behind its MMAs: the others arrive at its barriers and go on.
// Where there are CTAs for all SMs a CTA takes all of a head's value tiles, with the weights and the queries made once.
// Bound by the phases' latencies (one CTA an SM: 224 KB of shared memory, all of the tensor memory).
constexpr int OUT_NT = 512, OUT_ALL = OUT_NT + 32;
constexpr int TURN_LD = 20;                            // results on their way out: 32 rows of 16 a warp, padded by four
template <int NP> constexpr size_t out_smem() {
    return (size_t)(4 * (NP / 64) * ROWS_64 + 2 * ROWS_64 + 4 * NP * 128) + (NP == 128 ? 0 : OUT_NT * TURN_LD * 4) + 1024;
}
__device__ __forceinline__ void there(int i) { asm volatile("bar.arrive %0, %1;" ::"r"(i), "n"(OUT_ALL) : "memory"); }
__device__ __forceinline__ void all_there(int i) { asm volatile("bar.sync %0, %1;" ::"r"(i), "n"(OUT_ALL) : "memory"); }

template <int NP>
__global__ void __launch_bounds__(OUT_ALL, 1) decay_out_kernel(const DecayArgs a) {
    constexpr int PG = NP / 16, NB = NP / 64, TURNS = C * PG / OUT_NT;
    constexpr uint32_t ROWS_S = NP * 128;              // bytes of the state's rows of 64 columns
    constexpr uint32_t ID_QK = plm_tc::instr_desc_bf16(C), ID_MN = plm_tc::instr_desc_bf16(PT) | (1u << 16);
    constexpr uint32_t TM_W = 0, TM_P = 128, TM_STATE = 256, TM_O = 384;
    extern __shared__ uint8_t out_raw[];
    __shared__ uint64_t bars[3];
    __shared__ uint32_t slot;
    __shared__ float pw[C + 2];
    // of even and odd tiles: the first token that a column's odd values reach less 256 a tile (so that what a tile leaves is none of
    // the one after next), and one more than the last tile with any
    __shared__ int from[2][PT], any_odd[2];
    uint8_t* smem = out_raw + ((1024 - (plm_tc::smem_u32(out_raw) & 1023)) & 1023);
    uint8_t *qhi = smem, *qlo = qhi + NB * ROWS_64, *khi = qlo + NB * ROWS_64, *klo = khi + NB * ROWS_64, *vs = klo + NB * ROWS_64,
            *shi = vs + 2 * ROWS_64, *slo = shi + 2 * ROWS_S,
            *turn = NP == 128 ? khi : slo + 2 * ROWS_S;          // (the keys are done with when the first results are turned over)
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    pdl_launch_dependents();
    if (warp == 0) alloc_tmem(plm_tc::smem_u32(&slot), 512);
    const uint32_t bar = plm_tc::smem_u32(bars);
    if (tid == 0) {
        for (int i = 0; i < 3; ++i) plm_tc::mbar_init(bar + 8 * i, 1);
        any_odd[0] = any_odd[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_wait();
    const Where w = where_of(a);
    const int tiles = min(a.per, a.tiles - w.p0 / PT);
    if (tid < 2 * PT) (&from[0][0])[tid] = C;
    for (int i = tid; i <= C; i += OUT_ALL) pw[i] = power_of(a.powers + w.h * 65, i);
    plm_tc::tc_fence_before();
    __syncthreads();
    plm_tc::tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, slot, 0);
    if (w.n > 0 && warp == OUT_NT / 32) {
        const uint64_t qd[3] = {plm_tc::smem_desc_sw128(plm_tc::smem_u32(qlo)), plm_tc::smem_desc_sw128(plm_tc::smem_u32(qhi)),
                                plm_tc::smem_desc_sw128(plm_tc::smem_u32(qhi))};
        all_there(1);
        if (plm_tc::elect_one()) {                     // q . k, the smallest products first
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const uint64_t kd = plm_tc::smem_desc_sw128(plm_tc::smem_u32(i == 1 ? klo : khi));
#pragma unroll
                for (int s = 0; s < NP / 16; ++s) {
                    const uint32_t off = (s / 4 * ROWS_64 + s % 4 * 32) / 16;
                    plm_tc::tc_mma_bf16(tmem + TM_W, qd[i] + off, kd + off, ID_QK, i + s > 0);
                }
            }
            plm_tc::tc_commit(bar);
        }
        __syncwarp();
        for (int it = 0; it < tiles; ++it) {
            all_there(2);
            plm_tc::tc_fence_after();
            if (plm_tc::elect_one()) {                 // the state's share
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const uint64_t sd = desc_mn(plm_tc::smem_u32(i == 1 ? slo : shi), ROWS_S);
#pragma unroll
                    for (int s = 0; s < NP / 16; ++s)
                        plm_tc::tc_mma_bf16(tmem + TM_STATE, qd[i] + (s / 4 * ROWS_64 + s % 4 * 32) / 16, sd + s * 2048 / 16, ID_MN, i + s > 0);
                }
                plm_tc::tc_commit(bar + 8);
            }
            __syncwarp();
            if (it == 0) {
                all_there(3);
                plm_tc::tc_fence_after();
            }
            if (plm_tc::elect_one()) {
                const uint64_t vd = desc_mn(plm_tc::smem_u32(vs), ROWS_64);
#pragma unroll
                for (int term = 0; term < 2; ++term)
#pragma unroll
                    for (int s = 0; s < C / 16; ++s)
                        plm_split::mma_ts(tmem + TM_O, tmem + TM_P + (1 - term) * 64 + s * 8, vd + s * 2048 / 16, ID_MN, term + s > 0);
                plm_tc::tc_commit(bar + 16);
            }
            __syncwarp();
        }
    } else if (w.n > 0) {
        const long pos0 = a.half > 0 ? a.tok_pos[w.t0] : 0;
        const bf16* state = a.states + (a.slot(a.seq_start[w.b], w.b, w.c) * a.H + w.h) * 2l * NP * a.P + w.p0;
        auto load_tile = [&](int it) {                 // values and both terms of the state, straight to their places
            asm volatile("" ::: "memory");
#pragma unroll
            for (int i = 0; i < C * 16 / OUT_NT; ++i) {
                const int idx = tid + i * OUT_NT, r = idx / 16, c = idx % 16 * 8;
                const bool in = r < w.n;
                cp_async16(plm_tc::smem_u32(vs) + place(r, c), a.v + (long)(w.t0 + (in ? r : 0)) * a.ldv + (long)w.h * a.P + w.p0 + it * PT + c, in);
            }
#pragma unroll
            for (int i = 0; i < 2 * NP * 16 / OUT_NT; ++i) {
                const int idx = tid + i * OUT_NT, term = idx / (NP * 16), n = idx / 16 % NP, c = idx % 16 * 8;
                cp_async16(plm_tc::smem_u32(term ? slo : shi) + (uint32_t)(c >> 6) * ROWS_S + (uint32_t)n * 128 + ((((uint32_t)c >> 3) & 7) ^ ((uint32_t)n & 7)) * 16,
                           state + ((long)term * NP + n) * a.P + it * PT + c, true);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        load_tile(0);
        // (all loads of a batch before its first store: shared and global memory are one to the compiler)
        constexpr int BATCH = TURNS < 2 ? 1 : 2;
        static_assert(TURNS % BATCH == 0, "groups");
#pragma unroll
        for (int i0 = 0; i0 < TURNS; i0 += BATCH) {
            float4 cs[BATCH][4];
            uint4 x[BATCH][4];
#pragma unroll
            for (int i = 0; i < BATCH; ++i) {
                const int idx = tid + (i0 + i) * OUT_NT, r = idx / PG, g = idx % PG;
                const bool turn_it = g * 8 < a.half, in = r < w.n;
                const int cu = turn_it ? g * 8 : 2 * a.half + (g - a.half / 8) * 16, cv = turn_it ? a.half + g * 8 : cu + 8;
                x[i][0] = x[i][1] = x[i][2] = x[i][3] = make_uint4(0, 0, 0, 0);
                if (in) {
                    const bf16 *qr = a.q + (long)(w.t0 + r) * a.ldq + (long)w.h * NP, *kr = a.k + (long)(w.t0 + r) * a.ldk + (long)w.h * NP;
                    x[i][0] = *reinterpret_cast<const uint4*>(qr + cu), x[i][1] = *reinterpret_cast<const uint4*>(qr + cv);
                    x[i][2] = *reinterpret_cast<const uint4*>(kr + cu), x[i][3] = *reinterpret_cast<const uint4*>(kr + cv);
                }
                angles(a, pos0 + r, g * 8, turn_it && in, cs[i]);
            }
#pragma unroll
            for (int i = 0; i < BATCH; ++i) {
                const int idx = tid + (i0 + i) * OUT_NT, r = idx / PG, g = idx % PG;
                const bool turn_it = g * 8 < a.half;
                const int cu = turn_it ? g * 8 : 2 * a.half + (g - a.half / 8) * 16, cv = turn_it ? a.half + g * 8 : cu + 8;
                turn_to(x[i][0], x[i][1], turn_it, cs[i], 1.f, qhi, qlo, r, cu, cv);
                turn_to(x[i][2], x[i][3], turn_it, cs[i], a.k_scale, khi, klo, r, cu, cv);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        there(1);
        const int t = warp % 4 * 32 + lane, c0 = warp / 4 * 32;          // this thread's token and the first of its 32 columns
        const uint32_t lanes = tmem + ((uint32_t)(warp % 4 * 32) << 16);
        float* piece = reinterpret_cast<float*>(turn) + warp * 32 * TURN_LD;
        for (int it = 0; it < tiles; ++it) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
            for (int i = 0; i < C * 16 / OUT_NT; ++i) {              // what this thread has brought in of v
                const int idx = tid + i * OUT_NT, r = idx / 16, c = idx % 16 * 8;
                uint4 x = *reinterpret_cast<const uint4*>(vs + place(r, c));
                uint32_t* o = reinterpret_cast<uint32_t*>(&x);
                if (odd_one(o[0]) || odd_one(o[1]) || odd_one(o[2]) || odd_one(o[3])) {
                    any_odd[it & 1] = it + 1;
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const uint32_t half = o[e / 2] >> (16 * (e & 1)) & 0xffffu;
                        if ((half & 0x7f80u) == 0x7f80u) {
                            atomicMin(&from[it & 1][c + e], r - it * 256);
                            o[e / 2] &= e & 1 ? 0x0000ffffu : 0xffff0000u;
                        }
                    }
                    *reinterpret_cast<uint4*>(vs + place(r, c)) = x;
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            plm_tc::tc_fence_before();
            there(2);
            if (it == 0) {                             // the weights: a thread 32 of its token's
                plm_tc::mbar_wait_warp(bar, 0, a.status, 48);
                plm_tc::tc_fence_after();
                uint32_t hi[16], lo[16];
                if (c0 > warp % 4 * 32 + 31) {         // nothing that these tokens see
#pragma unroll
                    for (int j = 0; j < 16; ++j) hi[j] = lo[j] = 0;
                } else {
                    uint32_t r[32];
                    plm_split::tmem_load<32>(lanes + TM_W + c0, r);
                    plm_split::tmem_wait<32>(r);
#pragma unroll
                    for (int j = 0; j < 32; j += 2) {
                        const int d0 = t - (c0 + j), d1 = d0 - 1;
                        const float u = d0 >= 0 ? __uint_as_float(r[j]) * pw[max(d0, 0)] : 0.f, v = d1 >= 0 ? __uint_as_float(r[j + 1]) * pw[max(d1, 0)] : 0.f;
                        split2(u, v, hi[j / 2], lo[j / 2]);
                    }
                }
                store16(lanes + TM_P + c0 / 2, hi);
                store16(lanes + TM_P + 64 + c0 / 2, lo);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                plm_tc::tc_fence_before();
                there(3);
            }
            plm_tc::mbar_wait_warp(bar + 8, it & 1, a.status, 48);
            plm_tc::mbar_wait_warp(bar + 16, it & 1, a.status, 48);
            plm_tc::tc_fence_after();
            if (it + 1 < tiles) load_tile(it + 1);     // (what read the places is done)
            // turned over in shared memory, so that four lanes write 64 bytes in a row: a row a lane took 7,000 of a unit's 25,000 cycles
            const float d = pw[t + 1];
            const int odd = *(volatile int*)&any_odd[it & 1];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t r[16], o[16];
                plm_split::tmem_load<16>(lanes + TM_STATE + c0 + h * 16, r);
                plm_split::tmem_load<16>(lanes + TM_O + c0 + h * 16, o);
                plm_split::tmem_wait<16>(r);
                plm_split::tmem_wait<16>(o);
                __syncwarp();                          // (the piece before is read)
#pragma unroll
                for (int j = 0; j < 16; j += 4)
                    *reinterpret_cast<float4*>(piece + lane * TURN_LD + j) =
                        make_float4(fmaf(d, __uint_as_float(r[j]), __uint_as_float(o[j])), fmaf(d, __uint_as_float(r[j + 1]), __uint_as_float(o[j + 1])),
                                    fmaf(d, __uint_as_float(r[j + 2]), __uint_as_float(o[j + 2])), fmaf(d, __uint_as_float(r[j + 3]), __uint_as_float(o[j + 3])));
                __syncwarp();
                const int c = lane % 4 * 4, col = c0 + h * 16 + c;
                float* to = a.y + (long)w.t0 * a.ldy + (long)w.h * a.P + w.p0 + it * PT + col;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int row = i * 8 + lane / 4, tt = warp % 4 * 32 + row;
                    float4 v = *reinterpret_cast<const float4*>(piece + row * TURN_LD + c);
                    if (odd == it + 1) {
                        const float nan = __uint_as_float(0x7fffffffu);
                        auto reached = [&](int x) { const int f = from[it & 1][x] + it * 256; return f < C && tt >= f; };
                        if (reached(col)) v.x = nan;
                        if (reached(col + 1)) v.y = nan;
                        if (reached(col + 2)) v.z = nan;
                        if (reached(col + 3)) v.w = nan;
                    }
                    if (tt < w.n) *reinterpret_cast<float4*>(to + (long)tt * a.ldy) = v;
                }
            }
        }
    }
    plm_tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

template <int NP>
int launch(const DecayArgs& a, long places, cudaStream_t stream) {
    static std::atomic<unsigned long long> add_devices{0}, out_devices{0};
    static_assert(out_smem<NP>() <= 232448 - 1536, "shared memory");
    cudaError_t e = plm_allow_smem(decay_add_kernel<NP>, add_smem<NP>(), add_devices);
    if (e == cudaSuccess) e = plm_allow_smem(decay_out_kernel<NP>, out_smem<NP>(), out_devices);
    const dim3 units((unsigned)(places * a.H * ((a.tiles + a.per - 1) / a.per)));
    if (e == cudaSuccess) e = launch_pdl(decay_add_kernel<NP>, units, dim3(ADD_NT), add_smem<NP>(), stream, a);
    const long quads = (long)a.H * a.N * a.P / 4;
    if (e == cudaSuccess) e = launch_pdl(decay_states_kernel, dim3((unsigned)((quads + STATES_NT - 1) / STATES_NT), (unsigned)a.n_seqs), dim3(STATES_NT), 0, stream, a);
    if (e == cudaSuccess) e = launch_pdl(decay_out_kernel<NP>, units, dim3(OUT_ALL), out_smem<NP>(), stream, a);
    return plm_status_of(e);
}

}  // namespace

// Whether a step runs here, and the floats of workspace it takes (2 * (tokens / 128 + sequences) * H * N * P); 0: it
// runs in decay_chunk.cu.  At most 512 MB, as scan_chunk.cu takes (16 heads of 128 x 256: 16,000 tokens): a state for every chunk is
// more than that kernel's one for every segment.
extern "C" long plm_decay_tc_floats(int n_tokens, int n_seqs, int max_new, int H, int N, int P, int half) {
    if (n_seqs <= 0 || n_seqs > 65535 || max_new <= 0 || H <= 0 || (N != 64 && N != 128) || P <= 0 || P % PT || half % 8) return 0;
    const long floats = 2 * ((long)n_tokens / C + n_seqs) * H * N * P, units = ((long)n_tokens / C + n_seqs) * H * (P / PT);
    return floats <= (1l << 27) && units <= 0x7fffffffl ? floats : 0;
}

// q, k [T, H * N], v [T, H * P] bf16 with row strides (rows on 16-byte boundaries); powers [H][65] fp32; state [slots][>= H * N * P]
// fp32; y [T, H * P] fp32; ws of plm_decay_tc_floats floats; q and k are rotated (half pairs a head, cos and sin [positions][half]
// fp32, a sequence's positions consecutive from its first token's in tok_pos; half 0: not) and k times k_scale.
extern "C" int plm_decay_tc_scan(const void* q, const void* k, const void* v, long ldq, long ldk, long ldv, const float* powers, float* state,
                                 long state_stride, float* y, long ldy, const int* seq_start, const int* seq_slot, int n_tokens, int n_seqs,
                                 int max_new, int H, int N, int P, const float* cos_t, const float* sin_t, const int* tok_pos, int half,
                                 float k_scale, float* ws, int* status, cudaStream_t stream) {
    if (half < 0 || 2 * half > N || (half > 0 && (!cos_t || !sin_t || !tok_pos)) || !plm_decay_tc_floats(n_tokens, n_seqs, max_new, H, N, P, half))
        return PLM_ERR_SHAPE;
    if ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)state | (uintptr_t)y | (uintptr_t)ws | (uintptr_t)cos_t | (uintptr_t)sin_t) & 15) ||
        ldq % 8 || ldk % 8 || ldv % 8 || state_stride % 4 || ldy % 4)
        return PLM_ERR_ALIGN;
    DecayArgs a = {(const bf16*)q, (const bf16*)k, (const bf16*)v, ldq, ldk, ldv, powers, state, state_stride, y, ldy, seq_start, seq_slot,
                         n_seqs, H, N, P, cos_t, sin_t, tok_pos, half, k_scale, ws, (bf16*)(ws + ((long)n_tokens / C + n_seqs) * H * N * P), status, P / PT, 1};
    // a CTA takes all value tiles of its (chunk, head) where that leaves a CTA for most SMs
    const long places = (long)n_tokens / C + n_seqs;
    a.per = places * H >= PLM_SM_COUNT ? a.tiles : 1;
    return N == 64 ? launch<64>(a, places, stream) : launch<128>(a, places, stream);
}
