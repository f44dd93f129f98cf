// C[M,N] = A[M,K] * W[N,K]^T with fp32 accumulation on the CUDA cores.
//
// This is the reference's `matmul(out, x, W, n, d)`: W is row-major
// [out_features, in_features] and every output is the dot product of one weight
// row with the input (picolm/tensor.c:1394-1418), element types widened to fp32
// inside the dot product (picolm/quant.c:133-153, picolm/quant.c:679).
//
// It is the product of the float32 path where the weights are small (up to 131,072 of them) or rows do not start on
// 16-byte boundaries (the others run on the tensor cores, gemm_f32_tc.cu), of few-column pieces that a part asks for here,
// and the any-size product of the bfloat16 path when a shape does not fit the tensor-core kernel.  Each output element is accumulated over k in
// ascending order by one thread, so a row's result never depends on which other
// rows are in the batch.  With all three types float32 the sum of each piece of BK terms is folded into a
// double: the error of a long dot product then stays that of a short one (a recurrence that keeps a state for
// thousands of tokens multiplies what its gates' sums lose).
//
// With all three types float32 and rows that start on 16-byte boundaries, faster forms give the same bits: the sum of a
// piece of BK terms is the same chain of fused multiply-adds, and the pieces are folded into the double in the same
// order, so which form runs (it depends on the number of rows) shows in the time alone.
#include "common.cuh"
#include <type_traits>

namespace {

constexpr int BM = 64, BN = 64, BK = 16, NT = 256;

template <typename Ta, typename Tw, typename To>
__global__ void __launch_bounds__(NT)
gemm_simt_kernel(const Ta* A, const Tw* W, To* __restrict__ C, int M, int N, int K,
                 long lda, long ldw, long ldc) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int ty = tid / 16, tx = tid % 16;
    constexpr bool kWide = std::is_same<Ta, float>::value && std::is_same<Tw, float>::value && std::is_same<To, float>::value;
    float acc[4][4];
    double wide[kWide ? 4 : 1][kWide ? 4 : 1];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            acc[i][j] = 0.f;
            if (kWide) wide[kWide ? i : 0][kWide ? j : 0] = 0.0;
        }

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int it = 0; it < (BM * BK) / NT; ++it) {
            const int idx = tid + it * NT;
            const int r = idx / BK, k = idx % BK;
            const int gm = m0 + r, gn = n0 + r, gk = k0 + k;
            As[k][r] = (gm < M && gk < K) ? to_f32<Ta>(A[(size_t)gm * lda + gk]) : 0.f;
            Ws[k][r] = (gn < N && gk < K) ? to_f32<Tw>(W[(size_t)gn * ldw + gk]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Ws[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (kWide) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    wide[kWide ? i : 0][kWide ? j : 0] += (double)acc[i][j];
                    acc[i][j] = 0.f;
                }
        }
        __syncthreads();
    }
    if (kWide) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = (float)wide[kWide ? i : 0][kWide ? j : 0];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn < N) C[(size_t)gm * ldc + gn] = from_f32<To>(acc[i][j]);
        }
    }
}

// ---------------------------------------------------------------------------- float32, wide tiles
// Two fp32 lanes an instruction (fma.rn.f32x2 rounds each lane as fmaf does).
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

// A tile of TBM x TBN results, 8 x TN of them a thread (in pairs of rows), pieces of K turned over on their way into one
// of two buffers in shared memory while the other is read.
// Bound by the FMA pipe and by what stands between two pieces of K: without the folds (64 conversions and additions in
// double a thread and piece) the 64 x 128 form reaches 49.5 TFLOP/s of the pipe's 74, with them 38 at 512 rows x 16,384 x
// 2,048; the 64 x 64 form of 4 x 4 results a thread that ran before: 17 (462 x 16,384 x 2,048: 1,809 -> 894 us).  Two
// groups of threads a tile with every other piece each were no faster (204 against 187 us for a tile an SM), nor sums
// kept as pairs of floats (940 against 899).
template <int TBM, int TBN, int TN>
__global__ void __launch_bounds__((TBM / 8) * (TBN / TN))
gemm_f32_kernel(const float* A, const float* W, float* __restrict__ C, int M, int N, int K, long lda, long ldw, long ldc) {
    constexpr int TM = 8, TX = TBN / TN, TY = TBM / TM, THREADS = TX * TY, LDA = TBM + 4, LDB = TBN + 4;
    constexpr int QA = TBM * BK / 4 / THREADS, QB = TBN * BK / 4 / THREADS;          // float4 a thread brings in per piece
    static_assert(TX % 8 == 0 && TY % 4 == 0 && QA >= 1 && QB >= 1 && TN % 4 == 0, "tile");
    __shared__ __align__(16) float as[2][BK][LDA];
    __shared__ __align__(16) float bs[2][BK][LDB];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tx = lane % 8 + 8 * (warp % (TX / 8)), ty = lane / 8 + 4 * (warp / (TX / 8));
    const int m0 = blockIdx.y * TBM, n0 = blockIdx.x * TBN;
    const int q_row = tid / 4, q_k = (tid % 4) * 4;
    float4 ra[QA], rb[QB];
    auto fetch = [&](int k0) {
        const bool in_k = k0 + q_k < K;                                              // K is a multiple of 4
#pragma unroll
        for (int i = 0; i < QA; ++i) {
            const int m = m0 + q_row + i * (THREADS / 4);
            ra[i] = in_k && m < M ? *reinterpret_cast<const float4*>(A + (size_t)m * lda + k0 + q_k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < QB; ++i) {
            const int n = n0 + q_row + i * (THREADS / 4);
            rb[i] = in_k && n < N ? *reinterpret_cast<const float4*>(W + (size_t)n * ldw + k0 + q_k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto put = [&](int b) {
#pragma unroll
        for (int i = 0; i < QA; ++i) {
            const float v[4] = {ra[i].x, ra[i].y, ra[i].z, ra[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) as[b][q_k + j][q_row + i * (THREADS / 4)] = v[j];
        }
#pragma unroll
        for (int i = 0; i < QB; ++i) {
            const float v[4] = {rb[i].x, rb[i].y, rb[i].z, rb[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) bs[b][q_k + j][q_row + i * (THREADS / 4)] = v[j];
        }
    };
    double wide[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) wide[i][j] = 0.0;
    fetch(0);
    put(0);
    __syncthreads();
    int b = 0;
    for (int k0 = 0; k0 < K; k0 += BK, b ^= 1) {
        const bool more = k0 + BK < K;
        if (more) fetch(k0 + BK);
        uint64_t acc[TM / 2][TN];
#pragma unroll
        for (int i = 0; i < TM / 2; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = 0;                              // (0.f, 0.f)
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            uint64_t a2[TM / 2], b2[TN];
#pragma unroll
            for (int c = 0; c < TM / 4; ++c) {                                       // four rows of each half of the tile
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&as[b][k][c * (TY * 4) + ty * 4]);
                a2[2 * c] = v.x;
                a2[2 * c + 1] = v.y;
            }
#pragma unroll
            for (int c = 0; c < TN / 4; ++c) {
                const float4 v = *reinterpret_cast<const float4*>(&bs[b][k][c * (TX * 4) + tx * 4]);
                b2[4 * c] = pair_of(v.x, v.x);
                b2[4 * c + 1] = pair_of(v.y, v.y);
                b2[4 * c + 2] = pair_of(v.z, v.z);
                b2[4 * c + 3] = pair_of(v.w, v.w);
            }
#pragma unroll
            for (int i = 0; i < TM / 2; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fma2(a2[i], b2[j], acc[i][j]);
        }
        if (more) put(b ^ 1);
#pragma unroll
        for (int i = 0; i < TM / 2; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                float lo, hi;
                halves(acc[i][j], lo, hi);
                wide[2 * i][j] += (double)lo;
                wide[2 * i + 1][j] += (double)hi;
            }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + (i / 4) * (TY * 4) + ty * 4 + i % 4;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + (j / 4) * (TX * 4) + tx * 4 + j % 4;
            if (n < N) C[(size_t)m * ldc + n] = (float)wide[i][j];
        }
    }
}

// ---------------------------------------------------------------------------- float32, few rows
// A tile of FM rows x FN results.  Four pieces of K are worked on side by side by four groups of 64 threads; their sums
// meet in shared memory, where one thread a result folds them into its double in ascending order.  Rows arrive by
// cp.async, FSTAGES stages of four pieces deep.  Bound by the bytes in flight (24 rows x 2,048 x 8,192: 835 -> 111 us, 8
// rows: 833 -> 70 us; the weights alone take 10 at the copy rate).
constexpr int FK = 4 * BK, FLD = FK + 4, FSTAGES = 4;
template <int FM, int FN> constexpr size_t few_smem() { return (size_t)(FSTAGES * (FM + FN) * FLD + 2 * 4 * FM * FN) * sizeof(float); }

template <int FM, int FN>
__global__ void __launch_bounds__(256)
gemm_f32_few_kernel(const float* A, const float* W, float* __restrict__ C, int M, int N, int K, long lda, long ldw, long ldc) {
    constexpr int TM = FM / 8, TN = FN / 8, OUT = (FM * FN + 255) / 256;
    extern __shared__ __align__(16) float few[];
    float* sums = few + FSTAGES * (FM + FN) * FLD;                                   // [2][4][FM][FN]
    const int tid = threadIdx.x, group = tid / 64, tx = tid % 8, ty = tid / 8 % 8;
    const int m0 = blockIdx.y * FM, n0 = blockIdx.x * FN;
    const int n_stages = (K + FK - 1) / FK;
    auto fetch = [&](int s) {
        float* at = few + (s % FSTAGES) * (FM + FN) * FLD;
        for (int idx = tid; idx < (FM + FN) * (FK / 4); idx += 256) {
            const int row = idx / (FK / 4), k = s * FK + idx % (FK / 4) * 4;
            const bool is_a = row < FM;
            const int r = is_a ? m0 + row : n0 + row - FM;
            const bool in = k < K && r < (is_a ? M : N);                             // (outside: zeros, nothing is read)
            const float* src = in ? (is_a ? A + (size_t)r * lda + k : W + (size_t)r * ldw + k) : A;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(at + row * FLD + idx % (FK / 4) * 4)),
                         "l"(src), "r"(in ? 16 : 0) : "memory");
        }
    };
#pragma unroll
    for (int s = 0; s < FSTAGES - 1; ++s) {
        if (s < n_stages) fetch(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    double wide[OUT];
#pragma unroll
    for (int i = 0; i < OUT; ++i) wide[i] = 0.0;
    for (int s = 0; s < n_stages; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(FSTAGES - 2) : "memory");
        __syncthreads();                                    // stage s is there for all; stage s - 1 and the sums of s - 2 are read
        if (s + FSTAGES - 1 < n_stages) fetch(s + FSTAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* at = few + (s % FSTAGES) * (FM + FN) * FLD + group * BK;
        float acc[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 a[TM], w[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(at + (ty + 8 * i) * FLD + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(at + (FM + tx + 8 * j) * FLD + k);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j)
                    acc[i][j] = fmaf(a[i].w, w[j].w, fmaf(a[i].z, w[j].z, fmaf(a[i].y, w[j].y, fmaf(a[i].x, w[j].x, acc[i][j]))));
        }
        float* mine = sums + (s & 1) * 4 * FM * FN;
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) mine[(group * FM + ty + 8 * i) * FN + tx + 8 * j] = acc[i][j];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < OUT; ++i)
            if (tid + 256 * i < FM * FN)
#pragma unroll
                for (int p = 0; p < 4; ++p) wide[i] += (double)mine[p * FM * FN + tid + 256 * i];
    }
#pragma unroll
    for (int i = 0; i < OUT; ++i) {
        const int o = tid + 256 * i, m = m0 + o / FN, n = n0 + o % FN;
        if (o < FM * FN && m < M && n < N) C[(size_t)m * ldc + n] = (float)wide[i];
    }
}

template <int TBM, int TBN, int TN>
int launch_f32(const void* A, const void* W, void* C, int M, int N, int K, long lda, long ldw, long ldc, cudaStream_t stream) {
    gemm_f32_kernel<TBM, TBN, TN><<<dim3((N + TBN - 1) / TBN, (M + TBM - 1) / TBM), (TBM / 8) * (TBN / TN), 0, stream>>>(
        (const float*)A, (const float*)W, (float*)C, M, N, K, lda, ldw, ldc);
    return plm_launch_status();
}
template <int FM, int FN>
int launch_f32_few(const void* A, const void* W, void* C, int M, int N, int K, long lda, long ldw, long ldc, cudaStream_t stream) {
    static std::atomic<unsigned long long> devices{0};
    const cudaError_t configured = plm_allow_smem(gemm_f32_few_kernel<FM, FN>, few_smem<FM, FN>(), devices);
    if (configured != cudaSuccess) return (int)configured;
    gemm_f32_few_kernel<FM, FN><<<dim3((N + FN - 1) / FN, (M + FM - 1) / FM), 256, few_smem<FM, FN>(), stream>>>(
        (const float*)A, (const float*)W, (float*)C, M, N, K, lda, ldw, ldc);
    return plm_launch_status();
}

// The form whose waves of blocks take the least time: measured microseconds at K = 2,048 (all grow with K alike) of a wave with
// one, two or three blocks an SM, three or two being what an SM holds.
int f32_form(int M, int N) {
    struct Form { int bm, bn, per_sm, us[3]; };
    constexpr Form FORMS[] = {{8, 16, 3, {21, 29, 37}}, {32, 16, 3, {30, 43, 56}}, {32, 32, 2, {49, 72, 0}},
                              {64, 64, 3, {142, 170, 219}}, {64, 128, 2, {187, 258, 0}}};
    int best = 0;
    long best_us = -1;
    for (int f = 0; f < 5; ++f) {
        const Form& form = FORMS[f];
        const long rows = (M + form.bm - 1) / form.bm, blocks = rows * ((N + form.bn - 1) / form.bn);
        const long wave = (long)form.per_sm * PLM_SM_COUNT, rest = (blocks % wave + PLM_SM_COUNT - 1) / PLM_SM_COUNT;
        const long us = blocks / wave * form.us[form.per_sm - 1] + (rest ? form.us[rest - 1] : 0);
        if (rows <= 65535 && (best_us < 0 || us < best_us)) { best = f; best_us = us; }
    }
    return best;
}

// ---------------------------------------------------------------------------- bf16, few terms a sum
// out[t, n] for K of 8, 16 or 32 (a bottleneck's way back up): a thread keeps four columns' weights in registers and takes
// NARROW_ROWS rows, whose values it reads from shared memory.  Bound by the rows written.  The same chain of sums as
// gemm_simt_kernel (2,048 rows x 1,024 x 16: 7.8 -> 6.0 us without warm caches).
// With few results a thread's rows one behind the other take longer than that kernel's blocks side by side, so they go there.  us here /
// there, warm caches: 1 x 2,048 x 16 1.89 / 2.20, 4 x 2,048 x 32 3.09 / 3.50, 8 x 2,048 x 32 3.58 / 3.42, 64 x 2,048 x 16 3.25 / 2.74, 512 x
// 1,024 x 16 3.32 / 2.88, 256 x 4,096 x 16 3.32 / 3.94, 1,024 x 1,024 x 32 4.48 / 5.64, 4,096 x 256 x 16 4.27 / 3.70 (half of a block idles); 8
// terms: 16 x 1,024 2.55 / 2.48, 64 x 1,024 2.57 / 2.71, 2,048 x 1,024 3.18 / 5.94.
constexpr int NARROW_ROWS = 16;
template <int K>
__global__ void __launch_bounds__(128)
gemm_narrow_kernel(const bf16* A, const bf16* W, bf16* __restrict__ C, int M, int N, long lda, long ldw, long ldc) {
    __shared__ __align__(16) float as[NARROW_ROWS][K];
    const int m0 = blockIdx.y * NARROW_ROWS, n0 = (blockIdx.x * 128 + threadIdx.x) * 4;
    uint4 raw[4][K / 8];
    if (n0 < N)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < K / 8; ++i) raw[j][i] = *reinterpret_cast<const uint4*>(W + (size_t)(n0 + j) * ldw + i * 8);
#pragma unroll
    for (int i = threadIdx.x; i < NARROW_ROWS * K; i += 128) {
        const int r = i / K, k = i % K;
        as[r][k] = m0 + r < M ? to_f32<bf16>(A[(size_t)(m0 + r) * lda + k]) : 0.f;
    }
    __syncthreads();
    if (n0 >= N) return;
    float w[4][K];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < K / 8; ++i) {
            const uint32_t h[4] = {raw[j][i].x, raw[j][i].y, raw[j][i].z, raw[j][i].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                w[j][i * 8 + 2 * e] = __uint_as_float(h[e] << 16);
                w[j][i * 8 + 2 * e + 1] = __uint_as_float(h[e] & 0xffff0000u);
            }
        }
    for (int r = 0; r < NARROW_ROWS && m0 + r < M; ++r) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < K; k += 4) {
            const float4 a = *reinterpret_cast<const float4*>(&as[r][k]);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[j] = fmaf(a.w, w[j][k + 3], fmaf(a.z, w[j][k + 2], fmaf(a.y, w[j][k + 1], fmaf(a.x, w[j][k], acc[j]))));
        }
        const __nv_bfloat162 lo = __floats2bfloat162_rn(acc[0], acc[1]), hi = __floats2bfloat162_rn(acc[2], acc[3]);
        *reinterpret_cast<uint2*>(C + (size_t)(m0 + r) * ldc + n0) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
}

bool narrow_pays(int M, int N, int K) {
    return M <= 4 || (N >= 512 && (long)M * N >= (K == 8 ? 1l << 16 : 1l << 20));
}

template <int K>
int launch_narrow(const void* A, const void* W, void* C, int M, int N, long lda, long ldw, long ldc, cudaStream_t stream) {
    gemm_narrow_kernel<K><<<dim3((N + 511) / 512, (M + NARROW_ROWS - 1) / NARROW_ROWS), 128, 0, stream>>>((const bf16*)A, (const bf16*)W, (bf16*)C, M, N, lda, ldw, ldc);
    return plm_launch_status();
}

template <typename Ta, typename Tw, typename To>
int launch(const void* A, const void* W, void* C, int M, int N, int K, long lda, long ldw, long ldc,
           cudaStream_t stream) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    gemm_simt_kernel<Ta, Tw, To><<<grid, NT, 0, stream>>>((const Ta*)A, (const Tw*)W, (To*)C, M, N, K, lda, ldw, ldc);
    return plm_launch_status();
}

}  // namespace

// Leading dimensions are in elements.  Supported (A, W, C) element types:
// (f32,f32,f32), (bf16,bf16,bf16|f32), (bf16,f32,bf16|f32).
extern "C" int plm_gemm_simt(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype, int M, int N,
                             int K, long lda, long ldw, long ldc, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return PLM_OK;
    if (K <= 0 || lda < K || ldw < K || ldc < N) return PLM_ERR_SHAPE;
    if ((M + BM - 1) / BM > 65535) return PLM_ERR_SHAPE;
    if (a_dtype == PLM_F32 && w_dtype == PLM_F32 && c_dtype == PLM_F32 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
        !(((uintptr_t)A | (uintptr_t)W) & 15)) {
        const int best = f32_form(M, N);
        if (best == 0) return launch_f32_few<8, 16>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        if (best == 1) return launch_f32_few<32, 16>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        if (best == 2) return launch_f32_few<32, 32>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        if (best == 3) return launch_f32<64, 64, 4>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        return launch_f32<64, 128, 8>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    }
    if (a_dtype == PLM_F32 && w_dtype == PLM_F32 && c_dtype == PLM_F32)
        return launch<float, float, float>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    if (a_dtype == PLM_BF16 && w_dtype == PLM_BF16 && c_dtype == PLM_BF16 && (K == 8 || K == 16 || K == 32) && N % 4 == 0 && ldw % 8 == 0 &&
        ldc % 4 == 0 && (uintptr_t)W % 16 == 0 && (uintptr_t)C % 8 == 0 && (M + NARROW_ROWS - 1) / NARROW_ROWS <= 65535 && narrow_pays(M, N, K))
        return K == 8 ? launch_narrow<8>(A, W, C, M, N, lda, ldw, ldc, stream) : K == 16 ? launch_narrow<16>(A, W, C, M, N, lda, ldw, ldc, stream)
                                                                              : launch_narrow<32>(A, W, C, M, N, lda, ldw, ldc, stream);
    if (a_dtype == PLM_BF16 && w_dtype == PLM_BF16 && c_dtype == PLM_BF16)
        return launch<bf16, bf16, bf16>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    if (a_dtype == PLM_BF16 && w_dtype == PLM_BF16 && c_dtype == PLM_F32)
        return launch<bf16, bf16, float>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    if (a_dtype == PLM_BF16 && w_dtype == PLM_F32 && c_dtype == PLM_BF16)
        return launch<bf16, float, bf16>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    if (a_dtype == PLM_BF16 && w_dtype == PLM_F32 && c_dtype == PLM_F32)
        return launch<bf16, float, float>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    return PLM_ERR_DTYPE;
}

// Which of the float32 forms a product of M rows and N columns takes: 8 x 16, 32 x 16, 32 x 32 (few rows), 64 x 64, 64 x 128.
extern "C" int plm_gemm_simt_form(int M, int N) { return f32_form(M, N); }
