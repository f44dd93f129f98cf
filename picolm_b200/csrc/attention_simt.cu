// Causal attention of new tokens over the paged cache, one warp per
// (token, query head), on the CUDA cores with fp32 arithmetic throughout.
//
// For a query at absolute position p with head h, KV head g = h / (H / G):
//   s_t = (q_h . K[t, g]) * scale  for t in [lo, p],  out_h = softmax(s) . V[:, g]
// with the running (max, sum, acc) update of the reference's `attn_core`
// (picolm/model_attention.c:43-140; max starts at -1e30, causal by the loop
// bound) taken 32 keys at a time.  lo = 0, or p - window + 1 for a sliding
// window, or the start of p's chunk for a mask of chunks (plm_first_key); with `keep` > 0 the positions before
// min(keep, lo) are seen too; with `slopes` [H] a score loses slopes[h] * (p - t).  Keys and values of position t of sequence b live at
//   cache[block_table[b][t / PLM_PAGE]][g][t % PLM_PAGE][0..hd)
// and the new tokens' own K/V are already there when this kernel runs.
//
// This is the attention of the float32 path, and the any-size attention of the
// bfloat16 path (head sizes that the tensor-core kernels refuse).  A row's
// result depends on its own position and sequence only.
#include "common.cuh"

namespace {

constexpr int WARPS = 4;
constexpr int MAX_HD = 1024;           // the largest head size; acc registers per lane: MAX_HD / 32 of the instance

// MAX_HD: the instance's largest head size (256 for the usual heads; 512 and 1024 for the wide single head of a
// latent cache, whose keys are the latents themselves).
template <typename Ta, typename Tc, int MAX_HD>
__global__ void __launch_bounds__(WARPS * 32)
attention_rows_kernel(const Ta* q, const Tc* kc, const Tc* vc,
                      Ta* __restrict__ out, const int* tok_pos, const int* tok_seq,
                      const int* block_table, int max_pages, int H, int G, int hd, float scale,
                      int window, const float* sink, int keep, const float* slopes) {
    extern __shared__ float q_sm[];                 // [WARPS][hd]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x;
    const int h = blockIdx.y * WARPS + warp;
    if (h >= H) return;                             // warp-level exit; no block barrier below
    const int g = h / (H / G);
    const int pos = PLM_POSITION(tok_pos[t]);
    const int* pages = block_table + (size_t)PLM_SEQ_NO(tok_seq[t]) * max_pages;
    float* qs = q_sm + warp * hd;
    const Ta* qrow = q + ((size_t)t * H + h) * hd;
    for (int i = lane; i < hd; i += 32) qs[i] = to_f32<Ta>(qrow[i]);
    __syncwarp();

    float acc[MAX_HD / 32];
#pragma unroll
    for (int i = 0; i < MAX_HD / 32; ++i) acc[i] = 0.f;
    float m = -1e30f, l = 0.f;
    const int lo = plm_first_key(pos, window);
    const int n_kept = min(keep, lo);               // kept first positions in front of the window
    const int n_keys_all = n_kept + pos - lo + 1;
    const int skip = lo - n_kept;                   // the n-th key this row sees: n, or n + skip from n_kept on
    const float slope = slopes ? slopes[h] : 0.f;

    for (int base = 0; base < n_keys_all; base += 32) {
        const int nth = base + lane;
        const int key = nth < n_kept ? nth : nth + skip;
        float s = -1e30f;
        const bool valid = nth < n_keys_all;
        if (valid) {
            const int page = PLM_PAGE_NO(pages[key / PLM_PAGE]);
            const Tc* kr = kc + (((size_t)page * G + g) * PLM_PAGE + key % PLM_PAGE) * hd;
            float dot = 0.f;
            for (int i = 0; i < hd; ++i) dot = fmaf(qs[i], to_f32<Tc>(kr[i]), dot);
            s = __fmul_rn(dot, scale);
            if (slopes) s = fmaf(-slope, (float)(pos - key), s);
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float corr = expf(m - m_new);
        const float p = valid ? expf(s - m_new) : 0.f;
        l = fmaf(l, corr, warp_sum(p));
#pragma unroll
        for (int i = 0; i < MAX_HD / 32; ++i) acc[i] *= corr;
        const int n_keys = min(32, n_keys_all - base);
        for (int j = 0; j < n_keys; ++j) {
            const float pj = __shfl_sync(0xffffffffu, p, j);
            const int kj = base + j < n_kept ? base + j : base + j + skip;
            const int page = PLM_PAGE_NO(pages[kj / PLM_PAGE]);
            const Tc* vr = vc + (((size_t)page * G + g) * PLM_PAGE + kj % PLM_PAGE) * hd;
#pragma unroll
            for (int i = 0; i < MAX_HD / 32; ++i) {
                const int d = lane + 32 * i;
                if (d < hd) acc[i] = fmaf(pj, to_f32<Tc>(vr[d]), acc[i]);
            }
        }
        m = m_new;
    }
    if (sink) {
        // a sink: one more term exp(sink[h]) in the denominator, with no key and no value, not scaled
        const float sk = sink[h], m_new = fmaxf(m, sk);
        const float corr = expf(m - m_new);
        l = fmaf(l, corr, expf(sk - m_new));
#pragma unroll
        for (int i = 0; i < MAX_HD / 32; ++i) acc[i] *= corr;
    }
    const float inv = 1.0f / l;
    Ta* o = out + ((size_t)t * H + h) * hd;
#pragma unroll
    for (int i = 0; i < MAX_HD / 32; ++i) {
        const int d = lane + 32 * i;
        if (d < hd) o[d] = from_f32<Ta>(acc[i] * inv);
    }
}

// The same for prompts: a block takes 32 (token, query head) rows of one sequence and KV head, eight a warp, and brings the
// keys and values of 32 positions into shared memory once for all of them.  Without a mask every row's groups of 32 keys start
// at position 0, so a row sees the operations of the kernel above in the same order, bit for bit: how tokens are cut into
// steps does not show.  A sequence's tiles begin at block seq_start * (heads a KV head) / 32 + its number, so that single
// tokens beside a prompt have blocks of their own (tiles over several sequences walked their keys one after the other: 8
// tokens beside 63 single ones of 2,048 positions, 32 heads of 64, 1.9 ms by the kernel above, 12.3 by such tiles).
// Bound by shared memory (9 loads of 16 bytes for 32 multiply-adds); the kernel above reads every key's row from the
// second-level cache, a lane a row: 462 tokens of two sequences, 32 heads of 64 over 8, float32: 632 -> 75 us.
constexpr int TILE_ROWS = 32, ROWS_A_WARP = TILE_ROWS / WARPS;

template <typename T> __device__ __forceinline__ float4 load4(const T* p);
template <> __device__ __forceinline__ float4 load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 load4<bf16>(const bf16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                       __uint_as_float(v.y & 0xffff0000u));
}

static size_t tile_smem(int hd, int max_hd) { return (size_t)(32 * (hd + 4) + 32 * max_hd + TILE_ROWS * hd + TILE_ROWS * 32) * sizeof(float); }

template <typename T, int MAX_HD>
__global__ void __launch_bounds__(WARPS * 32)
attention_tile_kernel(const T* q, const T* kc, const T* vc, T* __restrict__ out, const int* tok_pos, const int* tok_seq,
                      const int* seq_start, int n_seqs, const int* block_table, int max_pages, int H, int G, int hd, float scale,
                      const float* sink, const float* slopes) {
    constexpr int VEC = MAX_HD / 32, R = ROWS_A_WARP;
    extern __shared__ __align__(16) float tile_sm[];
    float* ks = tile_sm;                            // [32][hd + 4]
    float* vs = ks + 32 * (hd + 4);                 // [32][MAX_HD], zero from hd on
    float* qs = vs + 32 * MAX_HD;                   // [TILE_ROWS][hd]
    float* ps = qs + TILE_ROWS * hd;                // [TILE_ROWS][32]
    __shared__ int warps_last[WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quads = hd / 4;
    const int per = H / G, g = blockIdx.y;
    // the sequence whose tiles this block is among: the last that begins at or before it
    int b = -1;
    for (int from = 0; from < n_seqs; from += WARPS * 32) {
        const int i = from + threadIdx.x;
        b += __syncthreads_count(i < n_seqs && (long)seq_start[i] * per / TILE_ROWS + i <= (long)blockIdx.x);
    }
    if (b < 0) return;
    const long tile = (long)blockIdx.x - ((long)seq_start[b] * per / TILE_ROWS + b);
    const long pair0 = (long)seq_start[b] * per + tile * TILE_ROWS, n_pairs = (long)seq_start[b + 1] * per;
    if (pair0 >= n_pairs) return;

    for (int i = threadIdx.x; i < TILE_ROWS * quads; i += WARPS * 32) {
        const long pair = pair0 + i / quads;
        const float4 v = pair < n_pairs ? load4<T>(q + ((pair / per) * H + g * per + pair % per) * hd + i % quads * 4)
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(qs + i / quads * hd + i % quads * 4) = v;
    }
    for (int i = threadIdx.x; i < 32 * (MAX_HD - hd); i += WARPS * 32) vs[i / (MAX_HD - hd) * MAX_HD + hd + i % (MAX_HD - hd)] = 0.f;

    float acc[R][VEC], m[R], l[R], slope[R];
    int tok[R], seen[R];                            // a row's token and position, -1 behind the sequence's last row
    int warp_last = -1, warp_first = 0x7fffffff;    // of the warp's rows: the largest and the smallest position
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const long pair = pair0 + warp * R + r;
        tok[r] = pair < n_pairs ? (int)(pair / per) : -1;
        seen[r] = tok[r] >= 0 ? PLM_POSITION(tok_pos[tok[r]]) : -1;
        warp_last = max(warp_last, seen[r]);
        warp_first = min(warp_first, seen[r]);
        slope[r] = slopes && tok[r] >= 0 ? slopes[g * per + pair % per] : 0.f;
        m[r] = -1e30f;
        l[r] = 0.f;
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[r][i] = 0.f;
    }
    if (lane == 0) warps_last[warp] = warp_last;
    const int* pages = block_table + (size_t)PLM_SEQ_NO(tok_seq[pair0 / per]) * max_pages;
    __syncthreads();
    int last_key = -1;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) last_key = max(last_key, warps_last[w]);
    for (int base = 0; base <= last_key; base += 32) {
        __syncthreads();                                             // what was there has been read (and q is there)
        for (int i = threadIdx.x; i < 32 * quads; i += WARPS * 32) {
            const int j = i / quads, c = i % quads * 4, key = base + j;
            float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), vv = kv;
            if (key <= last_key) {
                const size_t at = (((size_t)PLM_PAGE_NO(pages[key / PLM_PAGE]) * G + g) * PLM_PAGE + key % PLM_PAGE) * hd + c;
                kv = load4<T>(kc + at);
                vv = load4<T>(vc + at);
            }
            *reinterpret_cast<float4*>(ks + j * (hd + 4) + c) = kv;
            *reinterpret_cast<float4*>(vs + j * MAX_HD + c) = vv;
        }
        __syncthreads();
        if (base > warp_last) continue;
        float dot[R];
#pragma unroll
        for (int r = 0; r < R; ++r) dot[r] = 0.f;
        const float* kr = ks + lane * (hd + 4);
        const float* qr = qs + warp * R * hd;
#pragma unroll 2
        for (int i = 0; i < hd; i += 4) {
            const float4 kv = *reinterpret_cast<const float4*>(kr + i);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float4 qv = *reinterpret_cast<const float4*>(qr + r * hd + i);
                dot[r] = fmaf(qv.w, kv.w, fmaf(qv.z, kv.z, fmaf(qv.y, kv.y, fmaf(qv.x, kv.x, dot[r]))));
            }
        }
        float* pr = ps + warp * R * 32;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const bool valid = base + lane <= seen[r];
            float s = -1e30f;
            if (valid) {
                s = __fmul_rn(dot[r], scale);
                if (slopes) s = fmaf(-slope[r], (float)(seen[r] - base - lane), s);
            }
            const float m_new = fmaxf(m[r], warp_max(s));
            const float corr = expf(m[r] - m_new);
            const float p = valid ? expf(s - m_new) : 0.f;
            l[r] = fmaf(l[r], corr, warp_sum(p));
            m[r] = m_new;
#pragma unroll
            for (int i = 0; i < VEC; ++i) acc[r][i] *= corr;
            pr[r * 32 + lane] = p;
        }
        __syncwarp();
        const bool whole = warp_first >= base + 31;                  // every row sees all of the group's keys
#pragma unroll 2
        for (int j = 0; j < 32; j += 4) {
            float v[4][VEC];
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int i = 0; i < VEC; i += (VEC >= 4 ? 4 : 2)) {
                    const float* at = vs + (j + k) * MAX_HD + lane * VEC + i;
                    if (VEC >= 4) {
                        const float4 x = *reinterpret_cast<const float4*>(at);
                        v[k][i] = x.x; v[k][i + 1] = x.y; v[k][(i + 2) % VEC] = x.z; v[k][(i + 3) % VEC] = x.w;
                    } else {
                        const float2 x = *reinterpret_cast<const float2*>(at);
                        v[k][i] = x.x; v[k][i + 1] = x.y;
                    }
                }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float4 p4 = *reinterpret_cast<const float4*>(pr + r * 32 + j);
                const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (whole || base + j + k <= seen[r])            // (a value that a row does not see may be anything)
#pragma unroll
                        for (int i = 0; i < VEC; ++i) acc[r][i] = fmaf(p[k], v[k][i], acc[r][i]);
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (tok[r] < 0) continue;
        const int h = g * per + (int)((pair0 + warp * R + r) % per);
        if (sink) {
            const float sk = sink[h], m_new = fmaxf(m[r], sk);
            const float corr = expf(m[r] - m_new);
            l[r] = fmaf(l[r], corr, expf(sk - m_new));
#pragma unroll
            for (int i = 0; i < VEC; ++i) acc[r][i] *= corr;
        }
        const float inv = 1.0f / l[r];
        T* o = out + ((size_t)tok[r] * H + h) * hd;
#pragma unroll
        for (int i = 0; i < VEC; ++i)
            if (lane * VEC + i < hd) o[lane * VEC + i] = from_f32<T>(acc[r][i] * inv);
    }
}

}  // namespace

// q [T, H, hd] and out [T, H, hd] have the activation type, the cache its own;
// both are PLM_F32 or both PLM_BF16.  seq_start [n_seqs + 1] or null: where the step's sequences' rows begin.
extern "C" int plm_attention_rows(const void* q, const void* kc, const void* vc, void* out, int dtype,
                                  const int* tok_pos, const int* tok_seq, const int* block_table, int max_pages,
                                  int n_tokens, int H, int G, int hd, float scale, int window, const float* sink,
                                  int keep, const float* slopes, const int* seq_start, int n_seqs, cudaStream_t stream) {
    if (n_tokens <= 0) return PLM_OK;
    if (H <= 0 || G <= 0 || H % G || hd <= 0 || hd > MAX_HD || keep < 0) return PLM_ERR_SHAPE;
    // Prompts without a mask: tiles of a sequence's rows that share their keys (the caller says where that pays).
    if (seq_start && n_seqs > 0 && !window && !keep && hd % 4 == 0 && hd <= 256 && G <= 65535 &&
        !(((uintptr_t)q | (uintptr_t)kc | (uintptr_t)vc) & 15)) {
#define TILE_LAUNCH(T_, MAXHD_)                                                                                             \
    do {                                                                                                                    \
        static std::atomic<unsigned long long> devices{0};                                                                  \
        const cudaError_t configured = plm_allow_smem(attention_tile_kernel<T_, MAXHD_>, tile_smem(MAXHD_, MAXHD_), devices); \
        if (configured != cudaSuccess) return (int)configured;                                                              \
        const long pairs = (long)n_tokens * (H / G);                                                                        \
        attention_tile_kernel<T_, MAXHD_><<<dim3((unsigned)((pairs + TILE_ROWS - 1) / TILE_ROWS + n_seqs), G), WARPS * 32,            \
                                            tile_smem(hd, MAXHD_), stream>>>(                                               \
            (const T_*)q, (const T_*)kc, (const T_*)vc, (T_*)out, tok_pos, tok_seq, seq_start, n_seqs, block_table,     \
            max_pages, H, G, hd, scale, sink, slopes);                                                                      \
        return plm_launch_status();                                                                                         \
    } while (0)
#define TILE_BY_SIZE(T_)                     \
    do {                                     \
        if (hd <= 64) TILE_LAUNCH(T_, 64);   \
        if (hd <= 128) TILE_LAUNCH(T_, 128); \
        TILE_LAUNCH(T_, 256);                \
    } while (0)
        if (dtype == PLM_F32) TILE_BY_SIZE(float);
        if (dtype == PLM_BF16) TILE_BY_SIZE(bf16);
        return PLM_ERR_DTYPE;
#undef TILE_BY_SIZE
#undef TILE_LAUNCH
    }
    dim3 grid(n_tokens, (H + WARPS - 1) / WARPS);
    const size_t smem = (size_t)WARPS * hd * sizeof(float);
#define ROWS_LAUNCH(Ta_, MAXHD_)                                                                                       \
    attention_rows_kernel<Ta_, Ta_, MAXHD_><<<grid, WARPS * 32, smem, stream>>>(                                       \
        (const Ta_*)q, (const Ta_*)kc, (const Ta_*)vc, (Ta_*)out, tok_pos, tok_seq, block_table, max_pages, H, G, hd, \
        scale, window, sink, keep, slopes)
#define ROWS_BY_SIZE(Ta_)                          \
    do {                                           \
        if (hd <= 256) ROWS_LAUNCH(Ta_, 256);      \
        else if (hd <= 512) ROWS_LAUNCH(Ta_, 512); \
        else ROWS_LAUNCH(Ta_, 1024);               \
    } while (0)
    if (dtype == PLM_F32)
        ROWS_BY_SIZE(float);
    else if (dtype == PLM_BF16)
        ROWS_BY_SIZE(bf16);
    else
        return PLM_ERR_DTYPE;
#undef ROWS_BY_SIZE
#undef ROWS_LAUNCH
    return plm_launch_status();
}
