// Recurrences with a decay per key channel, for prompts, 64 tokens at a time in fp32:
//   linear attention   S <- diag(d_t) S + k_t v_t^T,                                   o_t = S^T q_t
//   the delta rule     S <- diag(d_t) S;  u_t = beta_t (v_t - S^T k_t);  S <- S + k_t u_t^T,  o_t = S^T q_t
// With S the state before a chunk, L_t the running sum of the decays' logarithms inside it (per head and key channel) and C
// its last token,
//   O = (q_t e^(L_t)) S + M U,          M_ts = sum_n q_tn k_sn e^(L_tn - L_sn), s <= t
//   S <- diag(e^(L_C)) S + sum_s (k_s e^(L_C - L_s)) u_s^T
// where U = V for linear attention, and for the delta rule the solution of a unit lower triangular system whose right side
// is linear in S:
//   U = U0 - W S,   (1 + A) U0 = (beta_t v_t),   (1 + A) W = (beta_t k_t e^(L_t)),   A_ts = beta_t sum_n k_tn k_sn e^(L_tn - L_sn), s < t
// Every exponent is <= 0: nothing is divided by a running decay, so no choice of decays overflows.
//
// What limits these is the chain from chunk to chunk, so only what needs the state stands in it.  All chunks side by side:
// the scaled keys and queries, M, A and both triangular systems (`chunk_prep`).  In a sequence's order: for the delta rule
// U and the state (`chunk_walk`, eight columns of the state a block), for linear attention a multiply and an add per value
// of the state (`chunk_chain`, behind every chunk's own sum of k u^T).  Then the outputs, all chunks side by side.  Those sums and
// the outputs are products on the tensor cores where the state has more than 64 columns (`chunk_product`), else FFMA tiles
// (`chunk_outer`, `chunk_out`); the rest runs on the CUDA cores.
// 2,048 tokens, 8 heads of 128 x 128, warm caches: the delta rule 518 us (32 tokens at a time, everything but the scaled keys and queries in
// the chain) -> 120, linear attention 144 us (token by token in segments) -> 65.  Errors against 64 bits in 2^-24, all products FFMA / on
// the tensor cores (512 tokens, 4 heads of 128 x 128, normal numbers; rows behind SiLU): linear attention's outputs 3.9 / 2.3 (2.8 / 1.4),
// state 2.5 / 1.5 (1.7 / 1.2), the delta rule's outputs 3.4 / 3.2 (2.6 / 2.4); where all values are positive and spread over several
// decades the tensor cores' are larger (3.3 / 4.2 and 1.8 / 3.0; see gemm_f32_tc.cu).
#include "split_common.cuh"
#include <type_traits>

namespace {

constexpr int C = 64;                    // tokens of a chunk
constexpr int B4 = 4, NB = C / B4, PAIRS = NB * (NB - 1) / 2;     // tokens of a block, blocks of a chunk (see chunk_prep)
constexpr int PREP_THREADS = 512;
constexpr int LDT = C + 4;               // a row of A^T in shared memory
constexpr int WALK_THREADS = 256, WC = 8;        // columns of the state a walking block keeps

struct Args {
    const void *q, *k, *v, *raw;         // rows of tokens; raw: the decays' logarithms (delta rule), or what makes them
    long ldq, ldk, ldv, ldr;
    const float *beta, *bias;            // delta rule: beta [T, H]; linear attention: bias [H, N] of the decay
    float power, q_scale;
    float* ws;
    float* state;
    long state_stride;
    float* y;                            // [T, H * P]
    const int *seq_start, *seq_slot;
    int H, N, P, heads_per_group, head_decay;
    int v_quads;                         // v's rows can be read four values at a time
    int* status;                         // device int that stays 0 unless a bounded wait ran out
    int b0, c0, stretch;                 // the launch's first sequence and chunk, and how many chunks of each sequence it takes (0: all)
    // the place in the workspace of a sequence's chunk: a whole step's chunks lie one behind the other, a stretch's by sequence
    __device__ long slot(int s0, int b, int c) const { return stretch ? (long)(b - b0) * stretch + (c - c0) : (long)(s0 / C + b + c); }
    __device__ int chunks_end(int n_chunks) const { return stretch ? min(n_chunks, c0 + stretch) : n_chunks; }
};

// The workspace of one (chunk, head), in floats.
// NP: the key size rounded up to 64 or 128, PP: the value size rounded up to a multiple of 4; padding is zero.
template <int NP> struct Layout {
    static constexpr long KE = 0, WT = KE + (long)C * NP, QT = WT + (long)C * NP, MT = QT + (long)C * NP, GE = MT + C * C, U = GE + NP;
    __host__ __device__ static long s(int PP) { return U + (long)C * PP; }           // the state that the chunk starts from
    __host__ __device__ static long floats(int PP) { return s(PP) + (long)NP * PP; }
};
__host__ __device__ inline int pad4(int P) { return (P + 3) / 4 * 4; }

__device__ __forceinline__ void cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void halves(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
template <typename T> __device__ __forceinline__ float4 quad(const T* p);
template <> __device__ __forceinline__ float4 quad<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 quad<bf16>(const bf16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                       __uint_as_float(v.y & 0xffff0000u));
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

template <int NP> constexpr size_t prep_smem() {
    return (size_t)(3 * C * (NP + 4) + C * LDT + NB * NP * 3 + PAIRS * NP + C) * sizeof(float);
}

// Everything of a chunk that does not depend on the state.  The exponentials of M and A would be one per pair of tokens and
// key channel; only pairs inside a block of four tokens take theirs.  For t in block I and s in an earlier block J,
//   e^(L_t - L_s) = e^(L_t - L_start(I)) e^(L_start(I) - L_end(J)) e^(L_end(J) - L_s)
// with three exponents <= 0: factors of t's row, of the pair of blocks, and of s's row.  Every exponent is a sum of
// logarithms and none a difference of running sums, where a strong decay's large sum would take the low digits of its
// neighbours' (2,048 tokens: 2.2e-6 off in the state with running sums, 2.2e-7 this way).
// Bound by shared memory (a float4 a lane is four of its cycles a warp), so products are tiles of 4 x 4 pairs of tokens a
// lane, with the channels dealt to four neighbouring lanes.  grid (chunk of the sequence, head, sequence: a captured
// step's sequences without tokens come last)
template <typename T, int NP, bool DELTA>
__global__ void __launch_bounds__(PREP_THREADS)
chunk_prep_kernel(const Args a) {
    constexpr int LD = NP + 4, SEG = C * NP / PREP_THREADS;
    static_assert(SEG % B4 == 0 && NB * 32 == PREP_THREADS && PAIRS * 4 <= PREP_THREADS && PAIRS * 4 % 32 == 0, "threads");
    using Lay = Layout<NP>;
    using Tk = typename std::conditional<DELTA, float, T>::type;         // the delta rule's q and k come in float32
    extern __shared__ __align__(16) float sm[];
    float* dec = sm;                     // [C][LD] the decays' logarithms; then k_s e^(L_end - L_s)
    float* ks = dec + C * LD;            // [C][LD] k; then k_t e^(L_t - L_start); then W, column by column
    float* qs = ks + C * LD;             // [C][LD] q; then q_t e^(L_t - L_start); then columns of U0
    float* At = qs + C * LD;             // [s][LDT], s < t
    float* tot = At + C * LDT;           // [NB][NP] sums over the blocks
    float* e_start = tot + NB * NP;      // [NB][NP] e^(L_start)
    float* e_rest = e_start + NB * NP;   // [NB][NP] e^(L_C - L_end)
    float* between = e_rest + NB * NP;   // [pairs of blocks I > J][NP] e^(L_start(I) - L_end(J))
    float* bt = between + PAIRS * NP;    // [C] beta, 0 behind the last token
    pdl_launch_dependents();
    pdl_wait();
    const int c = a.c0 + blockIdx.x, h = blockIdx.y, b = a.b0 + blockIdx.z, tid = threadIdx.x;
    const int s0 = a.seq_start[b], s1 = a.seq_start[b + 1], t0 = s0 + c * C;
    if (t0 >= s1) return;
    const int nt = min(C, s1 - t0), N = a.N, P = a.P, PP = pad4(P), H = a.H, g = h / a.heads_per_group;
    float* out = a.ws + (a.slot(s0, b, c) * H + h) * Lay::floats(PP);

    if (!DELTA) {                        // U is v
        const T* v = static_cast<const T*>(a.v) + (long)t0 * a.ldv + (long)h * P;
        if (a.v_quads) {
            for (int idx0 = tid; idx0 < C * (P / 4); idx0 += 8 * PREP_THREADS) {
                float4 vv[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int idx = idx0 + i * PREP_THREADS, t = min(idx / (P / 4), nt - 1), p = idx % (P / 4) * 4;
                    vv[i] = quad<T>(v + (long)t * a.ldv + p);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int idx = idx0 + i * PREP_THREADS;
                    if (idx < C * (P / 4)) *reinterpret_cast<float4*>(out + Lay::U + 4 * idx) = idx / (P / 4) < nt ? vv[i] : make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
        } else {
            for (int idx = tid; idx < C * PP; idx += PREP_THREADS) {
                const int t = idx / PP, p = idx % PP;
                out[Lay::U + idx] = t < nt && p < P ? to_f32<T>(v[(long)t * a.ldv + p]) : 0.f;
            }
        }
    }
    {   // keys, queries and the sums inside the blocks: a thread takes a channel's SEG tokens
        // (all loads are issued before the first is used: a load behind a condition would be waited for one by one, which
        // took 100 us of a 121 us kernel; places without a token or channel read a neighbour's and drop it)
        const int n = tid % NP, seg = tid / NP, nn = min(n, N - 1);
        const Tk* kp = static_cast<const Tk*>(a.k) + g * N + nn;
        const Tk* qp = static_cast<const Tk*>(a.q) + g * N + nn;
        Tk kv[SEG], qv[SEG];
        typename std::conditional<DELTA, float, T>::type rv[SEG];
        const auto* rp = static_cast<const typename std::conditional<DELTA, float, T>::type*>(a.raw) + (DELTA && a.head_decay ? h : h * N + nn);
#pragma unroll
        for (int i = 0; i < SEG; ++i) {
            const long row = t0 + min(seg * SEG + i, nt - 1);
            kv[i] = kp[row * a.ldk];
            qv[i] = qp[row * a.ldq];
            rv[i] = rp[row * a.ldr];
        }
        const float bias = DELTA ? 0.f : a.bias[h * N + nn];
        float run = 0.f;
#pragma unroll
        for (int i = 0; i < SEG; ++i) {
            const int t = seg * SEG + i;
            const bool in = t < nt && n < N;
            float l = to_f32<Tk>(rv[i]);
            if (!DELTA) {                // log(sigmoid(x)^power) = -power log(1 + e^(-x))
                const float x = l + bias;
                l = -a.power * (fmaxf(-x, 0.f) + log1pf(expf(-fabsf(x))));
            }
            if (!in) l = 0.f;
            run = i % B4 ? run + l : l;
            dec[t * LD + n] = l;
            ks[t * LD + n] = in ? to_f32<Tk>(kv[i]) : 0.f;
            qs[t * LD + n] = in ? to_f32<Tk>(qv[i]) * a.q_scale : 0.f;
            if (i % B4 == B4 - 1) tot[t / B4 * NP + n] = run;
        }
        if (DELTA && tid < C) bt[tid] = tid < nt ? a.beta[(long)(t0 + tid) * H + h] : 0.f;
    }
    __syncthreads();
    {   // a thread takes a channel and every GROUPS-th of the blocks that come first in a pair
        constexpr int GROUPS = PREP_THREADS / NP;
        const int n = tid % NP, group = tid / NP;
        float sums[NB];
#pragma unroll
        for (int j = 0; j < NB; ++j) sums[j] = tot[j * NP + n];
#pragma unroll
        for (int J = 0; J < NB - 1; ++J)
            if (J % GROUPS == group) {
                float run = 0.f;
#pragma unroll
                for (int I = J + 1; I < NB; ++I) {
                    between[(I * (I - 1) / 2 + J) * NP + n] = expf(run);
                    run += sums[I];
                }
                e_rest[J * NP + n] = expf(run);
            }
        if (group == GROUPS - 1) {
            float run = 0.f;
#pragma unroll
            for (int I = 0; I < NB; ++I) {
                e_start[I * NP + n] = expf(run);
                run += sums[I];
            }
            e_rest[(NB - 1) * NP + n] = 1.f;
            out[Lay::GE + n] = expf(run);
        }
    }
    const int warp = tid >> 5, lane = tid & 31;
    {   // pairs inside a block: a warp a block, a lane all of its pairs over four channels
        const int I = warp;
        float v[16];                     // A of (t, s) = 10 20 21 30 31 32; M of 00 10 11 20 21 22 30 31 32 33
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = 0.f;
        if (lane * 4 < NP) {
            float l[4][4], k[4][4], q[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int at = (I * B4 + i) * LD + lane * 4;
                *reinterpret_cast<float4*>(l[i]) = ld4(dec + at);
                *reinterpret_cast<float4*>(k[i]) = ld4(ks + at);
                *reinterpret_cast<float4*>(q[i]) = ld4(qs + at);
            }
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    float sum = 0.f;
#pragma unroll
                    for (int t = s; t < 4; ++t) {
                        if (t > s) sum += l[t][x];
                        const float e = t > s ? k[s][x] * expf(sum) : k[s][x];
                        v[6 + t * (t + 1) / 2 + s] = fmaf(q[t][x], e, v[6 + t * (t + 1) / 2 + s]);
                        if (s < t) v[t * (t - 1) / 2 + s] = fmaf(k[t][x], e, v[t * (t - 1) / 2 + s]);
                    }
                }
        }
#pragma unroll
        for (int half = 8, mask = 16; half >= 1; half >>= 1, mask >>= 1)         // lane 2 i (+ 1) ends with value i
#pragma unroll
            for (int i = 0; i < half; ++i) {
                const bool upper = (lane & mask) != 0;
                const float give = upper ? v[i] : v[i + half], keep = upper ? v[i + half] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, mask);
            }
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
        const int i = lane >> 1;
        if (!(lane & 1)) {
            const int j = i < 6 ? i : i - 6;
            int t = i < 6 ? 1 : 0, first = 0;                            // row t of the triangle starts at `first`
            while (first + t + (i < 6 ? 0 : 1) <= j) first += t + (i < 6 ? 0 : 1), ++t;
            const int s = j - first, tt = I * B4 + t, ss = I * B4 + s;
            if (i >= 6) out[Lay::MT + ss * C + tt] = v[0];
            else {
                if (DELTA) At[ss * LDT + tt] = bt[tt] * v[0];
                out[Lay::MT + tt * C + ss] = 0.f;                        // the pair the other way round
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NB * NP / PREP_THREADS; ++i) {                   // a thread a channel of a block
        const int idx = tid + i * PREP_THREADS, I = idx / NP, n = idx % NP, at = I * B4 * LD + n;
        const float rest = e_rest[I * NP + n];
        float d[B4], k[B4], run = 0.f;
#pragma unroll
        for (int t = 0; t < B4; ++t) {
            d[t] = dec[at + t * LD];
            k[t] = ks[at + t * LD];
            run += d[t];
            const float f = expf(run);
            ks[at + t * LD] = k[t] * f;
            qs[at + t * LD] *= f;
        }
        run = 0.f;
#pragma unroll
        for (int t = B4 - 1; t >= 0; --t) {
            const float hat = k[t] * expf(run);
            run += d[t];
            dec[at + t * LD] = hat;
            out[Lay::KE + (I * B4 + t) * NP + n] = hat * rest;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < C * NP / PREP_THREADS; ++i) {                    // the queries with the channels as rows
        const int idx = tid + i * PREP_THREADS, t = idx % C, n = idx / C;
        out[Lay::QT + idx] = qs[t * LD + n] * e_start[t / B4 * NP + n];
    }
    if (tid < PAIRS * 4) {               // pairs of blocks: four lanes a pair, each every fourth group of four channels
        const int u = tid >> 2, part = tid & 3;
        int I = 1;
        while (I * (I + 1) / 2 <= u) ++I;
        const int J = u - I * (I - 1) / 2;
        const float *d = between + u * NP, *kt = ks + I * B4 * LD, *qt = qs + I * B4 * LD, *hs = dec + J * B4 * LD;
        float x[4][4], m[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) x[i][j] = m[i][j] = 0.f;
        for (int n = part * 4; n < NP; n += 16) {
            const float4 dd = ld4(d + n);
            float4 hv[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                hv[j] = ld4(hs + j * LD + n);
                hv[j] = make_float4(hv[j].x * dd.x, hv[j].y * dd.y, hv[j].z * dd.z, hv[j].w * dd.w);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 kv = ld4(kt + i * LD + n), qv = ld4(qt + i * LD + n);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (DELTA) x[i][j] = fmaf(kv.w, hv[j].w, fmaf(kv.z, hv[j].z, fmaf(kv.y, hv[j].y, fmaf(kv.x, hv[j].x, x[i][j]))));
                    m[i][j] = fmaf(qv.w, hv[j].w, fmaf(qv.z, hv[j].z, fmaf(qv.y, hv[j].y, fmaf(qv.x, hv[j].x, m[i][j]))));
                }
            }
        }
        // the four lanes' sums: the first two end with A, the others with M, each with two of the four s (whole warps are here)
        float r[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float y[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float give = part & 2 ? x[i][j] : m[i][j];
                y[j] = (part & 2 ? m[i][j] : x[i][j]) + __shfl_xor_sync(0xffffffffu, give, 2);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float give = part & 1 ? y[j] : y[j + 2];
                r[i][j] = (part & 1 ? y[j + 2] : y[j]) + __shfl_xor_sync(0xffffffffu, give, 1);
            }
        }
        const int t = I * B4;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int s = J * B4 + (part & 1) * 2 + j;
            if (part & 2) *reinterpret_cast<float4*>(out + Lay::MT + s * C + t) = make_float4(r[0][j], r[1][j], r[2][j], r[3][j]);
            else if (DELTA)
                *reinterpret_cast<float4*>(At + s * LDT + t) = make_float4(bt[t] * r[0][j], bt[t + 1] * r[1][j], bt[t + 2] * r[2][j], bt[t + 3] * r[3][j]);
        }
        *reinterpret_cast<float4*>(out + Lay::MT + (t + part) * C + J * B4) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (!DELTA) return;
    __syncthreads();
    // Forward substitution, sixteen tokens at a time: a thread takes a column of the right sides, first those of W, then
    // those of U0, NP of either in a buffer; what is solved stays in the thread's column of the buffer for the tokens behind.
    for (int first = tid / NP; tid < 2 * NP && (first - 1) * NP < PP; first += 2) {
        const int n = tid % NP, p = (first - 1) * NP + n;
        const bool is_w = first == 0, in = is_w || p < P;
        float* buf = (tid < NP ? ks : qs) + n;
        const T* vc = static_cast<const T*>(a.v) + (long)t0 * a.ldv + (long)h * P + (in ? p : 0);
        if (!is_w && p >= PP) continue;
#pragma unroll 1
        for (int I = 0; I < C / 16; ++I) {
            float x[16];
            if (is_w) {
#pragma unroll
                for (int i = 0; i < 16; ++i) x[i] = bt[I * 16 + i] * buf[(I * 16 + i) * LD] * e_start[(I * 16 + i) / B4 * NP + n];
            } else {
                T vv[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) vv[i] = vc[(long)min(I * 16 + i, nt - 1) * a.ldv];
#pragma unroll
                for (int i = 0; i < 16; ++i) x[i] = in && I * 16 + i < nt ? bt[I * 16 + i] * to_f32<T>(vv[i]) : 0.f;
            }
#pragma unroll 4
            for (int s = 0; s < I * 16; ++s) {
                const float xs = buf[s * LD];
                const float* w = At + s * LDT + I * 16;
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const float4 y = ld4(w + i);
                    x[i] = fmaf(-y.x, xs, x[i]), x[i + 1] = fmaf(-y.y, xs, x[i + 1]);
                    x[i + 2] = fmaf(-y.z, xs, x[i + 2]), x[i + 3] = fmaf(-y.w, xs, x[i + 3]);
                }
            }
#pragma unroll
            for (int s = 0; s < 15; ++s) {
                const float* w = At + (I * 16 + s) * LDT + I * 16;
#pragma unroll
                for (int i = (s + 1) / 4 * 4; i < 16; i += 4) {
                    const float4 y = ld4(w + i);                         // (what lies at or before the diagonal is not used)
                    if (i > s) x[i] = fmaf(-y.x, x[s], x[i]);
                    if (i + 1 > s) x[i + 1] = fmaf(-y.y, x[s], x[i + 1]);
                    if (i + 2 > s) x[i + 2] = fmaf(-y.z, x[s], x[i + 2]);
                    x[i + 3] = fmaf(-y.w, x[s], x[i + 3]);
                }
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) buf[(I * 16 + i) * LD] = x[i];
            if (is_w) {
#pragma unroll
                for (int i = 0; i < 16; i += 4)
                    *reinterpret_cast<float4*>(out + Lay::WT + (long)n * C + I * 16 + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) out[Lay::U + (long)(I * 16 + i) * PP + p] = x[i];
            }
        }
    }
}

// One sequence's chunks in order, WC columns of the state a block: U = U0 - W S and the next state, both as small products
// whose long side is dealt to the warps and summed through shared memory.  The next chunk's W and keys arrive meanwhile.
// Bound by the chain (a chunk needs the one before; four barriers each) and by shared memory, about as much as by the FMA
// pipe (512 cycles a product): that is why a block keeps few columns and a head has P / WC of them.
// (a row of WC values of S or U starts four floats later for every four rows: neighbouring lanes write rows four apart)
__host__ __device__ constexpr int walk_row(int r) { return r * WC + r / 4 * 4; }
template <int NP> constexpr size_t walk_smem() { return (size_t)(2 * 2 * C * NP + walk_row(NP) + walk_row(C) + WALK_THREADS * 32) * sizeof(float); }

// acc[pair of rows][column] += rows (two pairs) x one row of WC values
__device__ __forceinline__ void outer_step(uint64_t (&acc)[2][WC], const float* rows, const float* cols) {
    const ulonglong2 r = *reinterpret_cast<const ulonglong2*>(rows);
    const float4 x = ld4(cols), y = ld4(cols + 4);
    const uint64_t v[WC] = {pair_of(x.x, x.x), pair_of(x.y, x.y), pair_of(x.z, x.z), pair_of(x.w, x.w),
                            pair_of(y.x, y.x), pair_of(y.y, y.y), pair_of(y.z, y.z), pair_of(y.w, y.w)};
#pragma unroll
    for (int j = 0; j < WC; ++j) acc[0][j] = fma2(r.x, v[j], acc[0][j]), acc[1][j] = fma2(r.y, v[j], acc[1][j]);
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

template <int NP, bool STRETCH>
__global__ void __launch_bounds__(WALK_THREADS)
chunk_walk_kernel(const Args a) {
    constexpr int NG = NP / 4, SPLITS = WALK_THREADS / NG, SS = C / SPLITS, NS = NP / 16, UNITS = 2 * NP;
    using Lay = Layout<NP>;
    extern __shared__ __align__(16) float sm[];
    float* Ss = sm + 2 * 2 * C * NP;     // [NP][WC]
    float* Us = Ss + walk_row(NP);       // [C][WC]
    float4* part = reinterpret_cast<float4*>(Us + walk_row(C));
    pdl_launch_dependents();
    const int P = a.P, PP = pad4(P), N = a.N, H = a.H, ptiles = (P + WC - 1) / WC;
    const int p0 = blockIdx.x % ptiles * WC, h = blockIdx.x / ptiles % H, b = (STRETCH ? a.b0 : 0) + blockIdx.x / ptiles / H;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_wait();
    const int s0 = a.seq_start[b], s1 = a.seq_start[b + 1];
    if (s1 <= s0) return;
    int n_chunks = (s1 - s0 + C - 1) / C;
    if (STRETCH) {                                     // from c0 on
        n_chunks = a.chunks_end(n_chunks) - a.c0;
        if (n_chunks <= 0) return;
    }
    const long step = (long)H * Lay::floats(PP);
    float* ws = a.ws + ((STRETCH ? a.slot(s0, b, a.c0) : (long)(s0 / C + b)) * H + h) * Lay::floats(PP);
    __shared__ __align__(8) uint64_t full[2];
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(full);
    if (tid == 0) {
        plm_tc::mbar_init(bar, 1);
        plm_tc::mbar_init(bar + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto fetch = [&](int chunk) {        // the scaled keys and W of a chunk lie side by side: one copy
        constexpr uint32_t BYTES = 2 * C * NP * sizeof(float);
        if (tid) return;
        const uint32_t at = bar + 8 * (chunk & 1);
        plm_tc::mbar_expect_tx(at, BYTES);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"((uint32_t)__cvta_generic_to_shared(sm + (chunk & 1) * 2 * C * NP)), "l"(ws + chunk * step + Lay::KE), "r"(BYTES), "r"(at)
                     : "memory");
    };
    fetch(0);
    // what this thread sums: four columns of one state row (threads below UNITS), four columns of one token (below 2 C)
    const int n = tid % NG * 4 + tid / NG / 2, cq = tid / NG % 2 * 4;
    const int ut = tid % 16 * 4 + tid / 16 % 2 * 2 + tid / 64, uq = tid / 32 % 2 * 4;
    const bool owns = tid < UNITS, owns_u = tid < 2 * C;
    float* st = a.state + (long)a.seq_slot[b] * a.state_stride + (long)h * N * P + (long)n * P + p0 + cq;
    float4 S = make_float4(0.f, 0.f, 0.f, 0.f);
    if (owns) {
        if (n < N) {
            if (p0 + cq < P) S.x = st[0];
            if (p0 + cq + 1 < P) S.y = st[1];
            if (p0 + cq + 2 < P) S.z = st[2];
            if (p0 + cq + 3 < P) S.w = st[3];
        }
        *reinterpret_cast<float4*>(Ss + walk_row(n) + cq) = S;
    }
    for (int chunk = 0; chunk < n_chunks; ++chunk) {
        float* w = ws + chunk * step;
        float4 u0 = make_float4(0.f, 0.f, 0.f, 0.f);
        const bool u_in = owns_u && p0 + uq < PP;
        float* u_at = w + Lay::U + (long)ut * PP + p0 + uq;
        if (u_in) u0 = ld4(u_at);
        const float ge = owns ? w[Lay::GE + n] : 0.f;
        if (owns && p0 + cq < PP) *reinterpret_cast<float4*>(w + Lay::s(PP) + (long)n * PP + p0 + cq) = S;
        // (a wait that runs out is noted and the walk goes on with what is there, so that no copy is in flight at the end)
        plm_tc::mbar_wait(bar + 8 * (chunk & 1), (chunk >> 1) & 1, a.status, 40);
        __syncthreads();
        if (chunk + 1 < n_chunks) fetch(chunk + 1);
        const float* ke = sm + (chunk & 1) * 2 * C * NP;
        const float* wt = ke + C * NP;
        {   // W S: sixteen shares of the channels, a lane four tokens
            uint64_t acc[2][WC] = {};
            const int tg = lane & 15, kh = lane >> 4, first = (warp * 2 + kh) * NS;
#pragma unroll
            for (int i = 0; i < NS; ++i) outer_step(acc, wt + (first + i) * C + tg * 4, Ss + walk_row(first + i));
            float lo[WC], hi[WC];                                        // the two half-warps trade a pair of tokens
#pragma unroll
            for (int j = 0; j < WC; ++j) {
                float mine_lo, mine_hi, give_lo, give_hi;
                halves(kh ? acc[1][j] : acc[0][j], mine_lo, mine_hi);
                halves(kh ? acc[0][j] : acc[1][j], give_lo, give_hi);
                lo[j] = mine_lo + __shfl_xor_sync(0xffffffffu, give_lo, 16);
                hi[j] = mine_hi + __shfl_xor_sync(0xffffffffu, give_hi, 16);
            }
            float4* at = part + warp * 128 + lane;
            at[0] = make_float4(lo[0], lo[1], lo[2], lo[3]);
            at[32] = make_float4(lo[4], lo[5], lo[6], lo[7]);
            at[64] = make_float4(hi[0], hi[1], hi[2], hi[3]);
            at[96] = make_float4(hi[4], hi[5], hi[6], hi[7]);
        }
        __syncthreads();
        if (owns_u) {
            float4 sum = part[tid];
#pragma unroll
            for (int i = 1; i < WALK_THREADS / 32; ++i) sum = add4(sum, part[i * 128 + tid]);
            u0 = make_float4(u0.x - sum.x, u0.y - sum.y, u0.z - sum.z, u0.w - sum.w);
            *reinterpret_cast<float4*>(Us + walk_row(ut) + uq) = u0;
            if (u_in) *reinterpret_cast<float4*>(u_at) = u0;
        }
        __syncthreads();
        {   // the keys times U: SPLITS shares of the tokens, a thread four channels
            uint64_t acc[2][WC] = {};
            const int ng = tid % NG, sp = tid / NG;
#pragma unroll
            for (int i = 0; i < SS; ++i) outer_step(acc, ke + (sp * SS + i) * NP + ng * 4, Us + walk_row(sp * SS + i));
            float4* at = part + sp * 8 * NG + ng;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float lo[WC], hi[WC];
#pragma unroll
                for (int j = 0; j < WC; ++j) halves(acc[i][j], lo[j], hi[j]);
                at[(4 * i) * NG] = make_float4(lo[0], lo[1], lo[2], lo[3]);
                at[(4 * i + 1) * NG] = make_float4(lo[4], lo[5], lo[6], lo[7]);
                at[(4 * i + 2) * NG] = make_float4(hi[0], hi[1], hi[2], hi[3]);
                at[(4 * i + 3) * NG] = make_float4(hi[4], hi[5], hi[6], hi[7]);
            }
        }
        __syncthreads();
        if (owns) {
            float4 sum = part[tid];
#pragma unroll
            for (int i = 1; i < SPLITS; ++i) sum = add4(sum, part[i * 8 * NG + tid]);
            S = make_float4(fmaf(ge, S.x, sum.x), fmaf(ge, S.y, sum.y), fmaf(ge, S.z, sum.z), fmaf(ge, S.w, sum.w));
            *reinterpret_cast<float4*>(Ss + walk_row(n) + cq) = S;
        }
    }
    if (owns && n < N) {
        if (p0 + cq < P) st[0] = S.x;
        if (p0 + cq + 1 < P) st[1] = S.y;
        if (p0 + cq + 2 < P) st[2] = S.z;
        if (p0 + cq + 3 < P) st[3] = S.w;
    }
}

// A tile of 64 rows x 64 columns of sums over rows of two row-major operands, A^T B, 16 rows of each at a time through a ring
// of three stages: `rows(step, a, b)` says where a step's rows start (a: 64 floats a row, b: 64 or as many as there are).
// 128 threads, 8 x 4 results each.
constexpr int TK = 16, TSTAGES = 3;
struct Tile {
    float a[TSTAGES][TK][64], b[TSTAGES][TK][64];
};
template <typename Rows>
__device__ __forceinline__ void tile_sums(Tile& tile, uint64_t (&acc)[4][4], int n_steps, int b_cols, Rows rows) {
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    auto fetch = [&](int i) {
        const float *pa, *pb;
        long lda, ldb;
        rows(i, pa, lda, pb, ldb);
        float* da = &tile.a[i % TSTAGES][0][0];
        float* db = &tile.b[i % TSTAGES][0][0];
#pragma unroll
        for (int x = 0; x < TK * 16 / 128; ++x) {
            const int idx = tid + 128 * x;
            cp16(da + idx * 4, pa + (idx / 16) * lda + idx % 16 * 4);
        }
#pragma unroll
        for (int x = 0; x < TK * 16 / 128; ++x) {
            const int idx = tid + 128 * x, col = idx % 16 * 4;
            if (col < b_cols) cp16(db + idx * 4, pb + (idx / 16) * ldb + col);
            else *reinterpret_cast<float4*>(db + idx * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
#pragma unroll
    for (int i = 0; i < TSTAGES - 1; ++i) {
        if (i < n_steps) fetch(i);
        cp_commit();
    }
    for (int i = 0; i < n_steps; ++i) {
        cp_wait<TSTAGES - 2>();
        __syncthreads();
        if (i + TSTAGES - 1 < n_steps) fetch(i + TSTAGES - 1);
        cp_commit();
        const int st = i % TSTAGES;
#pragma unroll
        for (int k = 0; k < TK; ++k) {
            uint64_t a2[4], b2[4];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&tile.a[st][k][x * 32 + ty * 4]);
                a2[2 * x] = v.x;
                a2[2 * x + 1] = v.y;
            }
            const float4 v = ld4(&tile.b[st][k][tx * 4]);
            b2[0] = pair_of(v.x, v.x);
            b2[1] = pair_of(v.y, v.y);
            b2[2] = pair_of(v.z, v.z);
            b2[3] = pair_of(v.w, v.w);
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[x][j] = fma2(a2[x], b2[j], acc[x][j]);
        }
    }
}
// the four columns tx * 4 .. of row r (0..7) of a thread's results
__device__ __forceinline__ float4 four(const uint64_t (&acc)[4][4], int r) {
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float lo, hi;
        halves(acc[r / 2][j], lo, hi);
        v[j] = r & 1 ? hi : lo;
    }
    return make_float4(v[0], v[1], v[2], v[3]);
}

// Linear attention: what a chunk adds to the state, sum_s (k_s e^(L_C - L_s)) v_s^T, into the state's place in the workspace.
// States of up to 64 columns; grid (chunk x channels by 64, head, sequence)
template <int NP>
__global__ void __launch_bounds__(128)
chunk_outer_kernel(const Args a) {
    using Lay = Layout<NP>;
    constexpr int MT = NP / 64;
    __shared__ __align__(16) Tile tile;
    pdl_launch_dependents();
    pdl_wait();
    const int PP = pad4(a.P), n0 = blockIdx.x % MT * 64, c = a.c0 + blockIdx.x / MT, h = blockIdx.y, b = a.b0 + blockIdx.z;
    const int s0 = a.seq_start[b], t0 = s0 + c * C, nt = min(C, a.seq_start[b + 1] - t0);
    if (nt <= 0) return;
    float* w = a.ws + (a.slot(s0, b, c) * a.H + h) * Lay::floats(PP);
    uint64_t acc[4][4] = {};
    tile_sums(tile, acc, (nt + TK - 1) / TK, PP, [&](int i, const float*& pa, long& lda, const float*& pb, long& ldb) {
        pa = w + Lay::KE + (long)i * TK * NP + n0, lda = NP;
        pb = w + Lay::U + (long)i * TK * PP, ldb = PP;
    });
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int n = n0 + r / 4 * 32 + ty * 4 + r % 4, p = tx * 4;
        if (p < PP)                                      // (padding stays zero, whatever U holds)
            *reinterpret_cast<float4*>(w + Lay::s(PP) + (long)n * PP + p) = n < a.N ? four(acc, r) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// Linear attention: the state at every chunk's start, a thread four columns of one channel; grid (NP * PP / 4 by 256, head, sequence)
template <int NP>
__global__ void __launch_bounds__(256)
chunk_chain_kernel(const Args a) {
    using Lay = Layout<NP>;
    constexpr int AHEAD = 8;
    pdl_launch_dependents();
    pdl_wait();
    const int P = a.P, PP = pad4(P), idx = blockIdx.x * 256 + threadIdx.x, h = blockIdx.y, b = a.b0 + blockIdx.z;
    const int n = idx / (PP / 4), p = idx % (PP / 4) * 4;
    const int s0 = a.seq_start[b], len = a.seq_start[b + 1] - s0;
    const int n_chunks = a.chunks_end((len + C - 1) / C) - a.c0;         // from c0 on
    if (n >= NP || n_chunks <= 0) return;
    const long step = (long)a.H * Lay::floats(PP);
    float* w = a.ws + (a.slot(s0, b, a.c0) * a.H + h) * Lay::floats(PP);
    float* at = w + Lay::s(PP) + (long)n * PP + p;
    float* st = a.state + (long)a.seq_slot[b] * a.state_stride + (long)h * a.N * P + (long)n * P + p;
    float4 S = make_float4(0.f, 0.f, 0.f, 0.f);
    if (n < a.N) {
        S.x = st[0];
        if (p + 1 < P) S.y = st[1];
        if (p + 2 < P) S.z = st[2];
        if (p + 3 < P) S.w = st[3];
    }
    for (int c0 = 0; c0 < n_chunks; c0 += AHEAD) {
        float4 add[AHEAD];
        float ge[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < n_chunks) add[i] = ld4(at + (c0 + i) * step), ge[i] = w[(c0 + i) * step + Lay::GE + n];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < n_chunks) {
                *reinterpret_cast<float4*>(at + (c0 + i) * step) = S;
                S = make_float4(fmaf(ge[i], S.x, add[i].x), fmaf(ge[i], S.y, add[i].y), fmaf(ge[i], S.z, add[i].z), fmaf(ge[i], S.w, add[i].w));
            }
    }
    if (n < a.N) {
        st[0] = S.x;
        if (p + 1 < P) st[1] = S.y;
        if (p + 2 < P) st[2] = S.z;
        if (p + 3 < P) st[3] = S.w;
    }
}

// O = Q S + M U of one chunk, for states of up to 64 columns; grid (chunk, head, sequence).  M is multiplied whole, zeros above its diagonal
// included; where a later token's row of U holds an infinity or no number, those products are no zeros, and a thread with a sum
// that comes out so takes its sums once more without them.  (Leaving them out of the tiles' steps, by steps and a select in the step on the
// diagonal, took 2 to 3 % of a mixer's time.)
template <int NP>
__global__ void __launch_bounds__(128)
chunk_out_kernel(const Args a) {
    using Lay = Layout<NP>;
    __shared__ __align__(16) Tile tile;
    pdl_launch_dependents();
    pdl_wait();
    const int P = a.P, PP = pad4(P), c = a.c0 + blockIdx.x, h = blockIdx.y, b = a.b0 + blockIdx.z;
    const int s0 = a.seq_start[b], t0 = s0 + c * C, nt = min(C, a.seq_start[b + 1] - t0);
    if (nt <= 0) return;
    const float* w = a.ws + (a.slot(s0, b, c) * a.H + h) * Lay::floats(PP);
    uint64_t acc[4][4] = {};
    tile_sums(tile, acc, NP / TK + (nt + TK - 1) / TK, PP, [&](int i, const float*& pa, long& lda, const float*& pb, long& ldb) {
        const int j = i - NP / TK;
        lda = C, ldb = PP;
        pa = w + (j < 0 ? Lay::QT + (long)i * TK * C : Lay::MT + (long)j * TK * C);
        pb = w + (j < 0 ? Lay::s(PP) + (long)i * TK * PP : Lay::U + (long)j * TK * PP);
    });
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    bool finite = true;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int t = r / 4 * 32 + ty * 4 + r % 4;
        if (t >= nt) continue;
        float* y = a.y + (long)(t0 + t) * a.H * P + (long)h * P;
        const int p = tx * 4;
        const float4 v = four(acc, r);
        if (p < P) finite = finite && fabsf(v.x) + fabsf(v.y) + fabsf(v.z) + fabsf(v.w) < INFINITY;
        if (P % 4 == 0) {
            if (p < P) *reinterpret_cast<float4*>(y + p) = v;
        } else {
            if (p < P) y[p] = v.x;
            if (p + 1 < P) y[p + 1] = v.y;
            if (p + 2 < P) y[p + 2] = v.z;
            if (p + 3 < P) y[p + 3] = v.w;
        }
    }
    if (!finite)                         // (rare: the same sums in the same order, over the rows that a token sees)
#pragma unroll 1
        for (int i = 0; i < 8 * 4; ++i) {
            const int t = i % 8 / 4 * 32 + ty * 4 + i % 4, p = tx * 4 + i / 8;
            if (t >= nt || p >= P) continue;
            float sum = 0.f;
#pragma unroll 1
            for (int n = 0; n < NP; ++n) sum = fmaf(w[Lay::QT + n * C + t], w[Lay::s(PP) + (long)n * PP + p], sum);
#pragma unroll 1
            for (int s = 0; s <= t; ++s) sum = fmaf(w[Lay::MT + s * C + t], w[Lay::U + (long)s * PP + p], sum);
            a.y[(long)(t0 + t) * a.H * P + (long)h * P + p] = sum;
        }
}

// The two products whose sides need no order between chunks, on the tensor cores: with OUT a chunk's O = Q S + M U, without it
// what a chunk of linear attention adds to the state, sum_s (k_s e^(L_C - L_s)) v_s^T.  A unit is one of these for 128 columns of
// the state: they are the MMA's rows, the chunk's tokens (or the state's channels) its columns, and the sums run over 32 rows of
// both operands at a time, every float in three bf16 terms as in gemm_f32_tc.cu.  Sums of pieces are added in fp32: the error
// against 64 bits is below that of the FFMA tiles, whose chains are six times as long.
// A CTA stays and walks over units; its warps' parts are those of gemm_f32_tc.cu, except that the operands come as plain bulk
// copies (their rows lie row by row in the workspace) and both are transposed on the way: a lane of the splitting warps reads one
// column's 32 rows for tensor memory, and the other operand stays as it lies, rows of 128 bytes with the 128-byte swizzle that
// the MMA reads with its N contiguous.
// Bound by the hand-overs between the warps, some 1,000 cycles a step (the tensor pipe is busy for 12 to 15 % of the time).  2,361 tokens in two
// sequences, 8 heads of 128 x 256, warm caches: outputs 47 us as FFMA tiles of 64 x 128 -> 31, what the chunks add 30 -> 21; 2,048
// tokens, 8 heads of 128 x 128: outputs 23.4 -> 14.5.
constexpr int TC_FOLDERS = 8, TC_LOADER = 16, TC_ISSUER = 17, TC_THREADS = 640, TC_RING = 4, TC_ROWS = 128, TC_STEP = 32;

template <int NB> struct TcTile {                                // NB columns of a unit: 64 or 128
    static constexpr int RAW_P = TC_STEP * TC_ROWS * 4, RAW = RAW_P + TC_STEP * NB * 4;
    static constexpr int BLOCK = TC_STEP * 128, TERM = NB / 64 * BLOCK, TERMS = 3 * TERM;
    static constexpr int TERMS_P = 2 * NB, TMEM = TERMS_P + 2 * 48 <= 256 ? 256 : 512;
    static constexpr size_t SMEM = TC_RING * RAW + 2 * TERMS + 1024;
};

// sums over the rows that a result depends on, one after the other (a result that is not finite: the split makes no numbers of
// infinities, and later tokens' zero weights make none of theirs)
template <int NP, bool OUT>
__device__ __noinline__ float sum_again(const float* w, int PP, int p, int col) {
    using Lay = Layout<NP>;
    float sum = 0.f;
    if (OUT) {
#pragma unroll 1
        for (int n = 0; n < NP; ++n) sum = fmaf(w[Lay::QT + n * C + col], w[Lay::s(PP) + (long)n * PP + p], sum);
#pragma unroll 1
        for (int s = 0; s <= col; ++s) sum = fmaf(w[Lay::MT + s * C + col], w[Lay::U + (long)s * PP + p], sum);
    } else {
#pragma unroll 1
        for (int s = 0; s < C; ++s) sum = fmaf(w[Lay::KE + s * NP + col], w[Lay::U + (long)s * PP + p], sum);
    }
    return sum;
}

template <int NP, bool OUT>
__global__ void __launch_bounds__(TC_THREADS, 1)
chunk_product_kernel(const __grid_constant__ CUtensorMap map_s, const __grid_constant__ CUtensorMap map_u, const Args a, int b_first, int chunks, int n_units) {
    using Lay = Layout<NP>;
    constexpr int NB = OUT ? C : NP, STEPS = OUT ? (NP + C) / TC_STEP : C / TC_STEP, R = TC_RING, COLS = NB / 2;
    using T = TcTile<NB>;
    // D fp32, A and B bf16, B with N contiguous
    constexpr uint32_t IDESC = plm_tc::instr_desc_bf16(NB) | (1u << 16);
    static_assert(R % 2 == 0 && STEPS % 2 == 0, "a splitting warp must not take a phase for the one after the next");
    static_assert(!OUT || STEPS >= 4, "a mark would stand where the unit before the last has not cleared its own");
    extern __shared__ unsigned char tc_raw[];
    __shared__ uint64_t bars[2 * R + 4];
    __shared__ uint32_t tmem_at;
    // OUT, of the even and of the odd units: the first token of the chunk that a column's values that are not finite reach (each
    // half of the adding warps has its own)
    constexpr int NOWHERE = 0x7fffffff;
    __shared__ int reached_from[2][2][TC_ROWS];
    unsigned char* smem = tc_raw + ((1024 - (plm_tc::smem_u32(tc_raw) & 1023)) & 1023);
    unsigned char* terms = smem + R * T::RAW;
    const uint32_t bar0 = plm_tc::smem_u32(bars);
    auto raw_full = [&](int b) { return bar0 + 8 * b; };
    auto raw_empty = [&](int b) { return bar0 + 8 * (R + b); };
    auto terms_full = [&](int b) { return bar0 + 8 * (2 * R + b); };
    auto mma_done = [&](int b) { return bar0 + 8 * (2 * R + 2 + b); };
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    pdl_launch_dependents();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(plm_tc::smem_u32(&tmem_at)), "r"(T::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int b = 0; b < R; ++b) {
            plm_tc::mbar_init(raw_full(b), 1);
            plm_tc::mbar_init(raw_empty(b), 4);
        }
        for (int b = 0; b < 2; ++b) {
            plm_tc::mbar_init(terms_full(b), 4 + TC_FOLDERS);    // the terms are there and the accumulator is read
            plm_tc::mbar_init(mma_done(b), 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < 4 * TC_ROWS) (&reached_from[0][0][0])[tid] = NOWHERE;
    plm_tc::tc_fence_before();
    __syncthreads();
    plm_tc::tc_fence_after();
    pdl_wait();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_at, 0);
    const int PP = pad4(a.P), ptiles = (PP + TC_ROWS - 1) / TC_ROWS;
    struct Unit { const float* w; int block, p0, h, t0, nt; };     // block: the (chunk, head)'s place in the workspace
    auto unit_at = [&](int u) {                                  // (nt <= 0: nothing there)
        Unit x;
        x.nt = 0;
        if (u >= n_units) return x;
        const unsigned v = (unsigned)u / (unsigned)ptiles, cb = v / (unsigned)chunks;
        x.p0 = (int)((unsigned)u - v * ptiles) * TC_ROWS;
        const int c = a.c0 + (int)(v - cb * chunks), b = b_first + (int)(cb / (unsigned)a.H), s0 = a.seq_start[b];
        x.h = (int)(cb % (unsigned)a.H);
        x.t0 = s0 + c * C;
        x.nt = min(C, a.seq_start[b + 1] - x.t0);
        x.block = (int)(a.slot(s0, b, c) * a.H + x.h);
        x.w = a.ws + x.block * Lay::floats(PP);
        return x;
    };
    // (a warp looks a unit up while it works on the one before)
    Unit next = unit_at(blockIdx.x);
    bool ok = true;
    int at = 0, turn = 0;                                        // steps so far, over all units; the unit's parity
    if (warp >= TC_LOADER) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        for (int u = blockIdx.x; u < n_units; u += gridDim.x) {
            const Unit x = next;
            next = unit_at(u + gridDim.x);
            if (x.nt <= 0) continue;
            if (warp == TC_LOADER) {
                for (int s = 0; s < STEPS; ++s, ++at) {
                    const int b = at % R;
                    if (at >= R) ok = ok && plm_tc::mbar_wait(raw_empty(b), ((at - R) / R) & 1, a.status, 44);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    const int j = s - NP / TC_STEP;              // OUT: Q and S first, then M and U
                    const bool first = OUT && j < 0;
                    const float* n_rows = OUT ? (j < 0 ? x.w + Lay::QT + (long)s * TC_STEP * C : x.w + Lay::MT + (long)j * TC_STEP * C)
                                              : x.w + Lay::KE + (long)s * TC_STEP * NP;
                    const uint32_t to = plm_tc::smem_u32(smem + b * T::RAW);
                    if (plm_tc::elect_one()) {
                        plm_tc::mbar_expect_tx(raw_full(b), T::RAW + PLM_STALL_BYTES);
                        asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                                     ::"r"(to), "l"((uint64_t)(first ? &map_s : &map_u)), "r"(raw_full(b)), "r"(x.p0),
                                       "r"((OUT && !first ? j : s) * TC_STEP), "r"(x.block) : "memory");
                        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                     ::"r"(to + T::RAW_P), "l"(n_rows), "r"(TC_STEP * NB * 4), "r"(raw_full(b)) : "memory");
                    }
                    __syncwarp();
                }
                if (!ok) break;
            } else if (warp == TC_ISSUER || warp == TC_ISSUER + 1) {         // every other step each, the smallest products first
                const int b = warp - TC_ISSUER;
                const uint32_t p = tmem + T::TERMS_P + b * 48, d = tmem + b * NB;
                const uint32_t n0 = plm_tc::smem_u32(terms + b * T::TERMS);
                // N contiguous: blocks of 64 columns BLOCK bytes apart, eight rows of K 1,024
                const uint64_t n = (uint64_t)((n0 & 0x3FFFFu) >> 4) | ((uint64_t)(T::BLOCK >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
                                   ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
                for (int s = (at ^ b) & 1; s < STEPS && ok; s += 2) {
                    ok = plm_tc::mbar_wait_warp(terms_full(b), ((at + s) >> 1) & 1, a.status, 45);
                    if (!ok) break;
                    plm_tc::tc_fence_after();
                    constexpr int TP[6] = {1, 2, 0, 1, 0, 0}, TN[6] = {1, 0, 2, 0, 1, 0};
                    if (plm_tc::elect_one()) {
#pragma unroll
                        for (int i = 0; i < 6; ++i)
#pragma unroll
                            for (int k = 0; k < TC_STEP / 16; ++k)
                                plm_split::mma_ts(d, p + TP[i] * 16 + k * 8, n + (TN[i] * T::TERM + k * 2048) / 16, IDESC, i + k > 0);
                        plm_tc::tc_commit(mma_done(b));
                    }
                    __syncwarp();
                }
                at += STEPS;
                if (!ok) break;
            }
        }
        if (warp == TC_LOADER)                                   // no copy may be under way when the CTA ends, whoever gave up
            for (int i = max(0, at - R); i < at; ++i) plm_tc::mbar_wait(raw_full(i % R), (i / R) & 1, nullptr, 0);
        __syncwarp();
    } else if (warp >= TC_FOLDERS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
        const int group = (warp - TC_FOLDERS) / 4, member = warp % 4;
        const uint32_t p_to = tmem + ((uint32_t)(member * 32) << 16) + T::TERMS_P + group * 48;
        unsigned char* n_to = terms + group * T::TERMS;
        for (int u = blockIdx.x; u < n_units && ok; u += gridDim.x) {
            const bool some = next.nt > 0;
            next = unit_at(u + gridDim.x);
            if (!some) continue;
            for (int s = group; s < STEPS; s += 2) {             // (a unit has an even number of steps)
                const int now = at + s, b = now % R;
                ok = plm_tc::mbar_wait_warp(raw_full(b), (now / R) & 1, a.status, 46);
                if (!ok) break;                                  // (a warp whose wait runs out arrives nowhere any more)
                const float* raw_p = reinterpret_cast<const float*>(smem + b * T::RAW) + member * 32 + lane;
                const float* raw_n = reinterpret_cast<const float*>(smem + b * T::RAW + T::RAW_P);
                int from = NOWHERE;
                uint32_t w[2][3][8];                             // (before the MMAs that read the buffers last are waited for)
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    float v[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = raw_p[(half * 16 + i) * TC_ROWS];
                    if (OUT) {
                        // A later token's weight is zero, but zero times what is not finite is not: such values go in as zeros, and
                        // the results of the tokens that see them are taken again, so that earlier ones stay as they are.
                        float check = 0.f;
#pragma unroll
                        for (int i = 0; i < 16; ++i) check = fmaf(v[i], 0.f, check);
                        if (!(check == 0.f))
#pragma unroll
                            for (int i = 0; i < 16; ++i)
                                if (!(fabsf(v[i]) < INFINITY)) {
                                    v[i] = 0.f;
                                    from = min(from, s < NP / TC_STEP ? 0 : (s - NP / TC_STEP) * TC_STEP + half * 16 + i);
                                }
                    }
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] *= plm_split::TERM_SCALE;
#pragma unroll
                    for (int t = 0; t < 3; ++t)
#pragma unroll
                        for (int i = 0; i < 8; ++i) w[half][t][i] = plm_split::next_terms(v[2 * i], v[2 * i + 1]);
                }
                if (now >= 2) ok = plm_tc::mbar_wait_warp(mma_done(group), ((now - 2) >> 1) & 1, a.status, 46);
                if (!ok) break;
                // (a mark's place is that of the unit before the last, whose marks must be read and cleared: behind this wait the
                // sums of step now - 4 are read, which is of the last unit where a unit has four steps)
                if (OUT && from != NOWHERE) {
                    atomicMin(&reached_from[turn][0][member * 32 + lane], from);
                    atomicMin(&reached_from[turn][1][member * 32 + lane], from);
                }
                __syncwarp();
                plm_tc::tc_fence_after();
#pragma unroll
                for (int half = 0; half < 2; ++half)
#pragma unroll
                    for (int t = 0; t < 3; ++t) plm_split::tmem_store8(p_to + t * 16 + half * 8, w[half][t]);
#pragma unroll
                for (int i = 0; i < TC_STEP * (NB / 8) / 128; ++i) {         // eight columns of a row
                    const int item = i * 128 + member * 32 + lane, k = item / (NB / 8), c8 = item % (NB / 8);
                    float v[8];
                    *reinterpret_cast<float4*>(v) = ld4(raw_n + k * NB + c8 * 8);
                    *reinterpret_cast<float4*>(v + 4) = ld4(raw_n + k * NB + c8 * 8 + 4);
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] *= plm_split::TERM_SCALE;
                    unsigned char* to = n_to + c8 / 8 * T::BLOCK + k * 128 + ((c8 % 8) ^ (k & 7)) * 16;
#pragma unroll
                    for (int t = 0; t < 3; ++t) {
                        uint4 x;
                        x.x = plm_split::next_terms(v[0], v[1]);
                        x.y = plm_split::next_terms(v[2], v[3]);
                        x.z = plm_split::next_terms(v[4], v[5]);
                        x.w = plm_split::next_terms(v[6], v[7]);
                        *reinterpret_cast<uint4*>(to + t * T::TERM) = x;
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                plm_tc::tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    plm_split::mbar_arrive(terms_full(group));
                    plm_split::mbar_arrive(raw_empty(b));
                }
            }
            at += STEPS;
            turn ^= 1;
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
        const uint32_t lanes = tmem + ((uint32_t)(warp % 4 * 32) << 16);
        const int c0 = warp / 4 * COLS;
        if (lane == 0) {                                         // both accumulators are free
            plm_split::mbar_arrive(terms_full(0));
            plm_split::mbar_arrive(terms_full(1));
        }
        __syncwarp();
        for (int u = blockIdx.x; u < n_units && ok; u += gridDim.x) {
            const Unit x = next;
            next = unit_at(u + gridDim.x);
            if (x.nt <= 0) continue;
            float sum[COLS];
#pragma unroll
            for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
#pragma unroll 1
            for (int s = 0; s < STEPS; ++s, ++at) {
                const int b = at & 1;
                ok = plm_tc::mbar_wait_warp(mma_done(b), (at >> 1) & 1, a.status, 47);
                if (PLM_GIVES_UP(warp, at)) {
                    atomicCAS(a.status, 0, 47);
                    ok = false;
                }
                if (!ok) break;
                plm_tc::tc_fence_after();
#pragma unroll
                for (int c = 0; c < COLS; c += 32) {
                    uint32_t r[32];
                    plm_split::tmem_load<32>(lanes + b * NB + c0 + c, r);
                    plm_split::tmem_wait<32>(r);
                    if (c + 32 == COLS) {
                        plm_tc::tc_fence_before();
                        __syncwarp();
                        if (lane == 0) plm_split::mbar_arrive(terms_full(b));
                    }
#pragma unroll
                    for (int j = 0; j < 32; ++j) sum[c + j] += __uint_as_float(r[j]);
                }
            }
            if (!ok) break;
            // (the stores first and what is not finite behind them: a look at each sum on its way out took 7,000 cycles a unit, more
            // than its six steps)
            const int p = x.p0 + warp % 4 * 32 + lane;
            const long ld = OUT ? (long)a.H * a.P : PP;
            float* to = OUT ? a.y + (long)(x.t0 + c0) * ld + (long)x.h * a.P + p : const_cast<float*>(x.w) + Lay::s(PP) + c0 * ld + p;
            const int rows = min(COLS, (OUT ? x.nt : a.N) - c0);
            bool finite = true;
            int from = NOWHERE;
            if (OUT) {
                int* mine = &reached_from[turn][warp / 4][warp % 4 * 32 + lane];
                from = *(volatile int*)mine;
                if (from != NOWHERE) *mine = NOWHERE;            // (the unit after next counts from there)
                turn ^= 1;
            }
            if (p < (OUT ? a.P : PP)) {
#pragma unroll
                for (int j = 0; j < COLS; ++j) {
                    if (!OUT && j >= rows) sum[j] = 0.f;         // (padding stays zero, whatever U holds)
                    if (!OUT || j < rows) {
                        finite = finite && fabsf(sum[j]) < INFINITY;
                        to[j * ld] = sum[j] * plm_split::SUM_SCALE;
                    }
                }
                if (!finite || from != NOWHERE)
#pragma unroll 1
                    for (int j = 0; j < rows; ++j)
                        if (c0 + j >= from || !(fabsf(to[j * ld]) < INFINITY)) to[j * ld] = sum_again<NP, OUT>(x.w, PP, p, c0 + j);
            }
            __syncwarp();
        }
        plm_tc::tc_fence_before();
    }
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::TMEM) : "memory");
}

// A workspace's rows of PP values, `rows` of them in every block of `block_floats`, as boxes of 32 rows x 128 columns (a copy of a
// row each, 33 a step, took three times the MMAs' time); kept by what they describe, as plm_tc::make_map's.
int make_rows_map(CUtensorMap* map, const float* first, int PP, int rows, long block_floats, long blocks) {
    struct Entry { const float* first; int PP, rows; long block_floats, blocks; bool used; CUtensorMap map; };
    constexpr int SLOTS = 64;
    static Entry table[SLOTS];
    static std::mutex lock;
    Entry& e = table[((((size_t)first >> 4) * 0x9E3779B97F4A7C15ull + (size_t)rows * 31 + (size_t)blocks * 131 + PP) >> 20) % SLOTS];
    {
        std::lock_guard<std::mutex> g(lock);
        if (e.used && e.first == first && e.PP == PP && e.rows == rows && e.block_floats == block_floats && e.blocks == blocks) {
            *map = e.map;
            return PLM_OK;
        }
    }
    plm_tc::EncodeTiledFn fn = plm_tc::encode_fn();
    if (!fn) return PLM_ERR_UNSUPPORTED;
    cuuint64_t dims[3] = {(cuuint64_t)PP, (cuuint64_t)rows, (cuuint64_t)blocks};
    cuuint64_t strides[2] = {(cuuint64_t)PP * 4, (cuuint64_t)block_floats * 4};
    cuuint32_t box[3] = {(cuuint32_t)TC_ROWS, (cuuint32_t)TC_STEP, 1}, estr[3] = {1, 1, 1};
    if (fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(first), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return PLM_ERR_ALIGN;
    std::lock_guard<std::mutex> g(lock);
    e.first = first; e.PP = PP; e.rows = rows; e.block_floats = block_floats; e.blocks = blocks; e.map = *map; e.used = true;
    return PLM_OK;
}

template <int NP, bool OUT>
int launch_product(const Args& a, long ws_floats, int n_seqs, unsigned chunks, cudaStream_t stream) {
    using Lay = Layout<NP>;
    static std::atomic<unsigned long long> devices{0};
    constexpr size_t SMEM = TcTile<OUT ? C : NP>::SMEM;
    static_assert(SMEM <= 232448 - 256, "shared memory");
    const cudaError_t ok = plm_allow_smem(chunk_product_kernel<NP, OUT>, SMEM, devices);
    if (ok != cudaSuccess) return (int)ok;
    const int PP = pad4(a.P);
    const long blocks = ws_floats / Lay::floats(PP), of_sequence = (long)chunks * ((PP + TC_ROWS - 1) / TC_ROWS) * a.H;
    CUtensorMap map_s, map_u;
    int r = make_rows_map(&map_s, a.ws + Lay::s(PP), PP, NP, Lay::floats(PP), blocks);
    if (r == PLM_OK) r = make_rows_map(&map_u, a.ws + Lay::U, PP, C, Lay::floats(PP), blocks);
    // (a launch's units, and a unit behind them, are counted in 32 bits: more of them take several launches)
    if (of_sequence > (1l << 30) || blocks > 0x7fffffffl) return PLM_ERR_SHAPE;
    const int at_once = (int)((1l << 30) / of_sequence < n_seqs ? (1l << 30) / of_sequence : n_seqs);
    for (int first = 0; r == PLM_OK && first < n_seqs; first += at_once) {
        const int units = (int)(of_sequence * (n_seqs - first < at_once ? n_seqs - first : at_once));
        r = plm_status_of(launch_pdl(chunk_product_kernel<NP, OUT>, dim3((unsigned)(units < PLM_SM_COUNT ? units : PLM_SM_COUNT)), dim3(TC_THREADS), SMEM,
                                     stream, map_s, map_u, a, a.b0 + first, (int)chunks, units));
    }
    return r;
}

template <int NP, bool STRETCH>
cudaError_t launch_walk(const Args& a, int n_seqs, cudaStream_t stream) {
    static std::atomic<unsigned long long> devices{0};
    const cudaError_t ok = plm_allow_smem(chunk_walk_kernel<NP, STRETCH>, walk_smem<NP>(), devices);
    if (ok != cudaSuccess) return ok;
    return launch_pdl(chunk_walk_kernel<NP, STRETCH>, dim3((unsigned)((long)n_seqs * a.H * ((a.P + WC - 1) / WC))), dim3(WALK_THREADS),
                      walk_smem<NP>(), stream, a);
}

template <int NP, typename T, bool DELTA, bool TC>
int run_stretch(const Args& a, long ws_floats, int n_seqs, unsigned chunks, cudaStream_t stream) {
    static std::atomic<unsigned long long> devices{0};
    const cudaError_t prep_ok = plm_allow_smem(chunk_prep_kernel<T, NP, DELTA>, prep_smem<NP>(), devices);
    if (prep_ok != cudaSuccess) return (int)prep_ok;
    if (!TC && a.P > 64) return PLM_ERR_SHAPE;                 // (the FFMA tiles have 64 columns)
    cudaError_t e = launch_pdl(chunk_prep_kernel<T, NP, DELTA>, dim3(chunks, a.H, n_seqs), dim3(PREP_THREADS), prep_smem<NP>(), stream, a);
    if (e != cudaSuccess) return (int)e;
    if (DELTA) {
        e = a.stretch ? launch_walk<NP, true>(a, n_seqs, stream) : launch_walk<NP, false>(a, n_seqs, stream);
    } else {
        if constexpr (TC) {
            const int r = launch_product<NP, false>(a, ws_floats, n_seqs, chunks, stream);
            if (r != PLM_OK) return r;
        } else
            e = launch_pdl(chunk_outer_kernel<NP>, dim3(chunks * (NP / 64), a.H, n_seqs), dim3(128), 0, stream, a);
        if (e != cudaSuccess) return (int)e;
        e = launch_pdl(chunk_chain_kernel<NP>, dim3((NP * (pad4(a.P) / 4) + 255) / 256, a.H, n_seqs), dim3(256), 0, stream, a);
    }
    if (e != cudaSuccess) return (int)e;
    if constexpr (TC) return launch_product<NP, true>(a, ws_floats, n_seqs, chunks, stream);
    else return plm_status_of(launch_pdl(chunk_out_kernel<NP>, dim3(chunks, a.H, n_seqs), dim3(128), 0, stream, a));
}

// The whole step at once where the workspace holds it.  Else so many chunks of so many sequences at a time as it holds: a state
// that a stretch leaves is what the next one starts from, as from step to step, so results are the same to the bit.
template <int NP, typename T, bool DELTA, bool TC>
int run(Args a, int n_tokens, int n_seqs, int max_new, long ws_floats, cudaStream_t stream) {
    const long chunks = (max_new + C - 1) / C, slots = ws_floats / (a.H * Layout<NP>::floats(pad4(a.P)));
    if ((long)n_tokens / C + n_seqs <= slots) return run_stretch<NP, T, DELTA, TC>(a, ws_floats, n_seqs, (unsigned)chunks, stream);
    if (slots < 1) return PLM_ERR_SHAPE;
    const int group = (int)(n_seqs < slots ? n_seqs : slots);
    a.stretch = (int)(slots / group < chunks ? slots / group : chunks);
    for (a.b0 = 0; a.b0 < n_seqs; a.b0 += group)
        for (a.c0 = 0; a.c0 < chunks; a.c0 += a.stretch) {
            const int e = run_stretch<NP, T, DELTA, TC>(a, ws_floats, n_seqs - a.b0 < group ? n_seqs - a.b0 : group, (unsigned)a.stretch, stream);
            if (e != PLM_OK) return e;
        }
    return PLM_OK;
}

template <typename T, bool DELTA>
int by_size(const Args& a, int n_tokens, int n_seqs, int max_new, long ws_floats, cudaStream_t stream) {
    // (a state of at most 64 columns would leave half of the MMA's rows idle: those run as FFMA tiles)
    if (a.N <= 64)
        return a.P <= 64 ? run<64, T, DELTA, false>(a, n_tokens, n_seqs, max_new, ws_floats, stream)
                         : run<64, T, DELTA, true>(a, n_tokens, n_seqs, max_new, ws_floats, stream);
    return a.P <= 64 ? run<128, T, DELTA, false>(a, n_tokens, n_seqs, max_new, ws_floats, stream)
                     : run<128, T, DELTA, true>(a, n_tokens, n_seqs, max_new, ws_floats, stream);
}

int check(const Args& a, int n_seqs, int max_new, int dtype) {
    if (a.H <= 0 || a.N <= 0 || a.P <= 0 || a.heads_per_group <= 0 || a.H % a.heads_per_group || n_seqs > 65535 || a.H > 65535) return PLM_ERR_SHAPE;
    if (a.N > 128) return PLM_ERR_UNSUPPORTED;
    if (dtype != PLM_F32 && dtype != PLM_BF16) return PLM_ERR_DTYPE;
    return PLM_OK;
}

}  // namespace

// Floats of workspace a (chunk, head) takes; a step of n_tokens tokens in n_seqs sequences runs at once in
// (n_tokens / 64 + n_seqs) * H of them, and in stretches in any number of H.
extern "C" int plm_scan_chunk_floats(int N, int P) { return (int)(N <= 64 ? Layout<64>::floats(pad4(P)) : Layout<128>::floats(pad4(P))); }

// The gated delta rule: qn, kn float32 [T, H / heads_per_group * N], dec (the decays' logarithms) float32 [T, H * N] or with
// head_decay [T, H], beta float32 [T, H], v of `dtype`; y float32 [T, H * P].
extern "C" int plm_delta_channel_scan(const float* qn, const float* kn, const float* dec, const float* beta, const void* v, int dtype,
                                      long ldv, float* state, long state_stride, float* y, float* ws, long ws_floats,
                                      const int* seq_start, const int* seq_slot, int n_tokens, int n_seqs, int max_new, int H, int N, int P,
                                      int heads_per_group, int head_decay, int* status, cudaStream_t stream) {
    if (n_seqs <= 0 || max_new <= 0) return PLM_OK;
    const long G = heads_per_group > 0 ? H / heads_per_group : 0;
    const Args a = {qn, kn, v, dec, G * N, G * N, ldv, head_decay ? (long)H : (long)H * N, beta, nullptr, 1.f, 1.f, ws, state, state_stride, y,
                    seq_start, seq_slot, H, N, P, heads_per_group, head_decay, 0, status, 0, 0, 0};
    const int e = check(a, n_seqs, max_new, dtype);
    if (e != PLM_OK) return e;
    return dtype == PLM_F32 ? by_size<float, true>(a, n_tokens, n_seqs, max_new, ws_floats, stream)
                            : by_size<bf16, true>(a, n_tokens, n_seqs, max_new, ws_floats, stream);
}

// Linear attention with the decays sigmoid(raw + bias)^power: q, k, v, raw of `dtype`.
extern "C" int plm_sigmoid_chunk_scan(const void* q, const void* k, const void* v, const void* raw, int dtype, long ldq, long ldk, long ldv,
                                      long ldr, const float* bias, float q_scale, float power, float* state, long state_stride, float* y,
                                      float* ws, long ws_floats, const int* seq_start, const int* seq_slot, int n_tokens, int n_seqs,
                                      int max_new, int H, int N, int P, int heads_per_group, int* status, cudaStream_t stream) {
    if (!bias) return PLM_ERR_SHAPE;
    if (n_seqs <= 0 || max_new <= 0) return PLM_OK;
    const Args a = {q, k, v, raw, ldq, ldk, ldv, ldr, nullptr, bias, power, q_scale, ws, state, state_stride, y, seq_start, seq_slot,
                    H, N, P, heads_per_group, 0,
                    P % 4 == 0 && ldv % 4 == 0 && (uintptr_t)v % (dtype == PLM_F32 ? 16 : 8) == 0, status, 0, 0, 0};
    const int e = check(a, n_seqs, max_new, dtype);
    if (e != PLM_OK) return e;
    return dtype == PLM_F32 ? by_size<float, false>(a, n_tokens, n_seqs, max_new, ws_floats, stream)
                            : by_size<bf16, false>(a, n_tokens, n_seqs, max_new, ws_floats, stream);
}
