// The experts' products of a routed feed-forward for prompts, bfloat16, on tcgen05: the chosen pairs' rows in sorted order
// (routed.cu, moe_align and moe_gather; an expert's rows start at a multiple of the sort's tile) times the expert's weights.
//
// The weights are the MMA's 128 rows and an expert's tokens its columns, up to 256 at once in steps of 16, so that no work is
// done for padding: with tokens on the 128 rows (what ran before), 192 rows an expert on average filled tiles of 128 to 60 %.
// What bounds it is then the weights' way from memory (537 MB of gate and up: 82 us), and what could stand in that way is the
// reading of the results (with one accumulator in turn, 43,000 of a unit's 69,000 cycles): so there are two, and eight warps
// read one while the next unit is under way.  A CTA an SM stays and takes units of 128 weight rows x an expert's tokens.  Warp 0
// loads (one tensor copy an operand and 64 of K, four stages; two stages of 128 of K took 123 us for 115), warp 1 issues the
// MMAs and owns the tensor memory; of the others each thread holds a weight row's results for 32 tokens, stored (or gated)
// from there.  With more rows an expert than some 224 the form with tokens on the rows is as fast again and stays.
// 2,048 tokens, 3 of 32 experts of 2,048 x 2,048 (gate and up, then down): 122 and 76 us -> 115 and 71 (4.9 and 4.7 of the
// 6.5 TB/s), and half as many rows to lay out in sorted order.
#include "tc_common.cuh"

using namespace plm_tc;

namespace {

// A test build only (-DPLM_TEST_GIVE_UP, never the library that serves): while the switch is 1, the loader announces 64 bytes
// more for every stage than it loads, so that every wait runs out; while it is 2, one warp of the eight that read results
// acts as if its wait for its CTA's second unit had run out.  The kernel must record it, let what it has in flight land, free
// its tensor memory and return.
#ifdef PLM_TEST_GIVE_UP
__device__ int plm_give_up_switch = 0;
#define PLM_STALL_BYTES (plm_give_up_switch == 1 ? 64u : 0u)
#define PLM_GIVES_UP(warp, unit) (plm_give_up_switch == 2 && (warp) == 3 && (unit) == 1)
#else
#define PLM_STALL_BYTES 0u
#define PLM_GIVES_UP(warp, unit) false
#endif

constexpr int FT = 128, EPI_WARPS = 8, THREADS = (2 + EPI_WARPS) * 32;
constexpr uint32_t W_SLAB = FT * 128, RING_BYTES = 196608;              // 64 of K of the weight rows; all stages
constexpr int MAX_GROUPS = 1024;
constexpr uint32_t TURN = 2 * 16 * 64 * 4;             // what the gate's and the up branch's threads hand each other, an accumulator
constexpr size_t SMEM = (size_t)RING_BYTES + 2 * TURN + 1024 + 256;
enum { STORE = 0, GATED = 1, RELU2 = 2 };

// Whether all 128 threads of a named barrier say yes.
__device__ __forceinline__ bool set_agrees(int barrier, bool yes) {
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.and.pred q, %2, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(all) : "r"(yes ? 1u : 0u), "r"(barrier) : "memory");
    return all != 0;
}

struct Unit { int row, n, f0, group; };                // first sorted row, its tokens (a multiple of 16), first weight row, expert

// NMAX: the most tokens of a unit; SLABS: how many times 64 of K a copy brings in, lying one behind the other.
template <int EPI, typename OutT, int NMAX, int SLABS>
__global__ void __launch_bounds__(THREADS, 1)
moe_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x64, const __grid_constant__ CUtensorMap map_x128,
              const __grid_constant__ CUtensorMap map_x192, const __grid_constant__ CUtensorMap map_x256, OutT* __restrict__ out, long ldo,
              const int* tile_expert, int max_tiles, int bm, int E, int F, int K, int* status) {
    constexpr uint32_t W_BYTES = SLABS * W_SLAB, STAGE = W_BYTES + SLABS * NMAX * 128;
    constexpr int RING = RING_BYTES / STAGE;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ int first_tile[MAX_GROUPS], last_tile[MAX_GROUPS], units_before[MAX_GROUPS + 1];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_abort;
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    const uint32_t turn0 = base + RING_BYTES, full0 = turn0 + 2 * TURN, empty0 = full0 + 8 * RING, acc_full0 = empty0 + 8 * RING,
                   acc_empty0 = acc_full0 + 16;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_launch_dependents();
    if (tid == 0) {
        s_abort = 0;
        for (int s = 0; s < RING; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(acc_full0 + 8 * s, 1); mbar_init(acc_empty0 + 8 * s, EPI_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int e = tid; e < E; e += THREADS) { first_tile[e] = 0; last_tile[e] = -1; }
    pdl_wait();
    __syncthreads();
    for (int i = tid; i < max_tiles; i += THREADS) {   // the tiles of one expert are neighbours
        const int e = tile_expert[i];
        if (e < 0) continue;
        if (i == 0 || tile_expert[i - 1] != e) first_tile[e] = i;
        if (i + 1 == max_tiles || tile_expert[i + 1] != e) last_tile[e] = i;
    }
    __syncthreads();
    const int f_tiles = (F + FT - 1) / FT;
    if (warp == 0) {                                   // (32 experts at a time: one by one, 1,024 of them took some 25 us a launch)
        int before = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane;
            int sum = e < E ? ((last_tile[e] - first_tile[e] + 1) * bm + NMAX - 1) / NMAX * f_tiles : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int below = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += below;
            }
            if (e < E) units_before[e + 1] = before + sum;
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) units_before[0] = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const int n_units = units_before[E], n_k = (K + SLABS * BK - 1) / (SLABS * BK);
    // Unit u: experts in order, an expert's tokens in equal chunks, a chunk's weight rows one after the other (neighbouring CTAs
    // share the tokens, and every weight row is read once a chunk).
    auto unit_at = [&](int u) {
        int lo = 0, hi = E;                            // the last e with units_before[e] <= u (and units of its own)
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (units_before[mid] <= u) lo = mid; else hi = mid;
        }
        const int rows = (last_tile[lo] - first_tile[lo] + 1) * bm, chunks = (rows + NMAX - 1) / NMAX;
        const int per = (rows / chunks + 15) / 16 * 16, in = u - units_before[lo], chunk = in / f_tiles;
        Unit x;
        x.group = lo;
        x.row = first_tile[lo] * bm + chunk * per;
        x.n = min(per, rows - chunk * per);
        x.f0 = in % f_tiles * FT;
        return x;
    };

    if (warp == 0) {
        // ------------------------------------------------------------ tensor copies
        if (lane == 0) {
            int i = 0;
            for (int u = blockIdx.x; u < n_units; u += gridDim.x) {
                const Unit x = unit_at(u);
                const int box = (x.n + 63) / 64;
                const CUtensorMap* map_x = box == 1 ? &map_x64 : box == 2 ? &map_x128 : box == 3 ? &map_x192 : &map_x256;
                for (int k = 0; k < n_k; ++k, ++i) {
                    const uint32_t bar = full0 + 8 * (i % RING), dst = base + (i % RING) * STAGE;
                    if (*(volatile int*)&s_abort || !mbar_wait(empty0 + 8 * (i % RING), ((i / RING) & 1) ^ 1, status, 51)) { s_abort = 1; break; }
                    mbar_expect_tx(bar, W_BYTES + SLABS * box * 64 * 128 + PLM_STALL_BYTES);
                    if (SLABS > 1) {
                        tma_load_3d(dst, &map_w, bar, x.group * F + x.f0, k * SLABS);
                        tma_load_3d(dst + W_BYTES, map_x, bar, x.row, k * SLABS);
                    } else {
                        tma_load_2d(dst, &map_w, bar, k * BK, x.group * F + x.f0);
                        tma_load_2d(dst + W_BYTES, map_x, bar, k * BK, x.row);
                    }
                }
                if (*(volatile int*)&s_abort) break;
            }
            if (*(volatile int*)&s_abort)              // let what is in flight land
                for (int s = max(0, i - RING); s < i; ++s) mbar_wait(full0 + 8 * (s % RING), (s / RING) & 1, nullptr, 0);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMAs
        if (elect_one()) {
            int i = 0, done = 0, handed = 0;           // stages consumed, units begun, units handed to the warps that read them
            bool ok = true;
            for (int u = blockIdx.x; u < n_units && ok; u += gridDim.x, ++done) {
                const Unit x = unit_at(u);
                const uint32_t idesc = instr_desc_bf16(x.n), x_slab = (x.n + 63) / 64 * 64 * 128;
                const int acc = done & 1;
                if (!mbar_wait(acc_empty0 + 8 * acc, ((done >> 1) & 1) ^ 1, status, 52)) { ok = false; break; }
                tc_fence_after();
                for (int k = 0; k < n_k; ++k, ++i) {
                    if (*(volatile int*)&s_abort || !mbar_wait(full0 + 8 * (i % RING), (i / RING) & 1, status, 53)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t w = base + (i % RING) * STAGE, t = w + W_BYTES;
#pragma unroll
                    for (int s = 0; s < SLABS; ++s)
#pragma unroll
                        for (int j = 0; j < BK / UMMA_K; ++j)
                            tc_mma_bf16(tmem + acc * NMAX, smem_desc_sw128(w + s * W_SLAB) + (uint64_t)(j * 2),
                                        smem_desc_sw128(t + s * x_slab) + (uint64_t)(j * 2), idesc, (k > 0 || s > 0 || j > 0) ? 1u : 0u);
                    tc_commit(empty0 + 8 * (i % RING));
                }
                if (ok) { tc_commit(acc_full0 + 8 * acc); ++handed; }
            }
            if (!ok) s_abort = 1;
            // what was issued has to be done, and its commits to have arrived, before the tensor memory and the barriers go
            for (int s = max(0, i - RING); s < i; ++s) mbar_wait(empty0 + 8 * (s % RING), (s / RING) & 1, nullptr, 0);
            for (int x = max(0, handed - 2); x < handed; ++x) mbar_wait(acc_full0 + 8 * (x & 1), (x >> 1) & 1, nullptr, 0);
        }
    } else {
        // ------------------------------------------------------------ results: two sets of four warps, 32 tokens in turn
        const int set = (warp - 2) / 4, quarter = warp & 3, r = quarter * 32 + lane;     // this thread's weight row of the 128
        const bool up = r >= 64;
        float* turn = reinterpret_cast<float*>(smem_raw + (turn0 + set * TURN - raw));   // [2][16 tokens][64]
        float* give = turn + (up ? 0 : 16 * 64) + (r & 63);
        const float* take = turn + (up ? 16 * 64 : 0) + (r & 63);
        int done = 0;
        for (int u = blockIdx.x; u < n_units; u += gridDim.x, ++done) {
            const Unit x = unit_at(u);
            const int acc = done & 1, f = EPI == GATED ? x.f0 / 2 + (r & 63) : x.f0 + r;
            const bool in_f = f < (EPI == GATED ? F / 2 : F);
            const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + acc * NMAX;
            // One verdict for all that meet below: the lanes of a warp (tcgen05.ld), and with a gate the four warps of a set (the
            // barriers around what they hand each other have no limit of their own).
            bool there = mbar_wait_warp(acc_full0 + 8 * acc, (done >> 1) & 1, status, 54);
            if (PLM_GIVES_UP(warp, done)) { atomicCAS(status, 0, 54); there = false; }
            if (EPI == GATED) there = set_agrees(1 + set, there);
            if (!there) { s_abort = 1; break; }
            tc_fence_after();
            for (int c = set * 32; c < x.n; c += 64) {
                uint32_t v[32];
                tc_ld32(at + c, v);                    // (behind the n columns that were written: not used)
                tc_wait_ld_into(v);
                const bool second = c + 16 < x.n;      // (n is a multiple of 16)
                OutT* to = out + (size_t)(x.row + c) * ldo + f;
                if (EPI == GATED) {
                    // rows 0..63 are the gate's, 64..127 the up branch's: each side hands the other sixteen tokens
#pragma unroll
                    for (int j = 0; j < 16; ++j) give[j * 64] = __uint_as_float(up ? v[j] : v[16 + j]);
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory");
                    if (in_f && (!up || second)) {
                        if (up) to += 16 * ldo;
#pragma unroll
                        for (int j = 0; j < 16; ++j, to += ldo) {
                            const float mine = __uint_as_float(up ? v[16 + j] : v[j]), other = take[j * 64];
                            *to = from_f32<OutT>(swiglu_bf16(up ? other : mine, up ? mine : other));
                        }
                    }
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory");
                } else if (in_f) {
#pragma unroll
                    for (int j = 0; j < 32; ++j, to += ldo) {
                        float z = __uint_as_float(v[j]);
                        if (EPI == RELU2) {
                            z = fmaxf(z, 0.f);
                            z *= z;
                        }
                        if (j < 16 || second) *to = from_f32<OutT>(z);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty0 + 8 * acc) : "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

template <int EPI, typename OutT, int NMAX, int SLABS>
int launch_form(const void* x, const void* w, void* out, long ldo, const int* tile_expert, int max_tiles, int bm, int E, int F, int K, int* status,
                cudaStream_t stream) {
    auto kernel = moe_tc_kernel<EPI, OutT, NMAX, SLABS>;
    static std::atomic<unsigned long long> devices{0};
    const cudaError_t configured = plm_allow_smem(kernel, SMEM, devices);
    if (configured != cudaSuccess) return (int)configured;
    CUtensorMap m[5];
    int rc = make_map(&m[0], w, (long)E * F, K, K, FT, SLABS);
    for (int i = 1; i < 5 && rc == PLM_OK; ++i)            // tokens 64, 128, 192 or 256 at a time
        rc = make_map(&m[i], x, (long)max_tiles * bm, K, K, 64 * i < NMAX ? 64 * i : NMAX, SLABS);
    if (rc != PLM_OK) return rc;
    return plm_status_of(launch_pdl(kernel, dim3(PLM_SM_COUNT), dim3(THREADS), SMEM, stream, m[0], m[1], m[2], m[3], m[4], (OutT*)out, ldo,
                                    tile_expert, max_tiles, bm, E, F, K, status));
}

template <int EPI, typename OutT>
int launch(const void* x, const void* w, void* out, long ldo, int n_pairs, const int* tile_expert, int max_tiles, int bm, int E, int F, int K,
           int* status, cudaStream_t stream) {
    // Experts with some 100 rows or fewer on average: 128 tokens at once leave room for three stages of 128 of K.  A copy keeps
    // its SM's copy engine for some 190 cycles and 6.6 a KB, and with few tokens that is longer than the MMAs of 64 of K.
    // 32 experts of 2,048 x 2,048 with 19, 66 and 91 rows each: 154, 167 and 175 us for a layer against 168, 181 and 189 in the
    // other form; with 122 rows 196 against 197 and with 192, in two parts, 261 against 226.
    if (K % BK == 0 && n_pairs <= 104 * E)
        return launch_form<EPI, OutT, 128, 2>(x, w, out, ldo, tile_expert, max_tiles, bm, E, F, K, status, stream);
    return launch_form<EPI, OutT, 256, 1>(x, w, out, ldo, tile_expert, max_tiles, bm, E, F, K, status, stream);
}

}  // namespace

// out[row, :] = f(x[row, :] W[tile_expert[row / bm]]^T) for the rows of all tiles that have an expert (the tiles of one expert
// are neighbours; bm a multiple of 16; n_pairs: how many rows the tiles hold, which chooses a form).  x [rows, K] bf16, w
// [E, F, K] bf16.  epilogue 0: store (fp32), 1: gate and up rows in turns of 64, silu(gate) * up (out [rows, F / 2] bf16),
// 2: squared ReLU (bf16).
// `status`: a device int that stays 0 unless a bounded wait ran out.
extern "C" int plm_moe_tc(const void* x, const void* w, void* out, int out_dtype, int epilogue, int n_pairs, const int* tile_expert,
                          int max_tiles, int bm, int E, int F, int K, long ldo, int* status, cudaStream_t stream) {
    if (max_tiles <= 0) return PLM_OK;
    if (E <= 0 || F <= 0 || K < BK || bm <= 0 || bm % 16 || ldo < (epilogue == GATED ? F / 2 : F)) return PLM_ERR_SHAPE;
    if (E > MAX_GROUPS || K % 8 || (epilogue == GATED && F % 128)) return PLM_ERR_UNSUPPORTED;
    if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out) & 15) return PLM_ERR_ALIGN;
    if (epilogue == GATED || epilogue == RELU2) {
        if (out_dtype != PLM_BF16) return PLM_ERR_DTYPE;
        return epilogue == GATED ? launch<GATED, bf16>(x, w, out, ldo, n_pairs, tile_expert, max_tiles, bm, E, F, K, status, stream)
                                 : launch<RELU2, bf16>(x, w, out, ldo, n_pairs, tile_expert, max_tiles, bm, E, F, K, status, stream);
    }
    if (epilogue != STORE) return PLM_ERR_UNSUPPORTED;
    if (out_dtype != PLM_F32) return PLM_ERR_DTYPE;
    return launch<STORE, float>(x, w, out, ldo, n_pairs, tile_expert, max_tiles, bm, E, F, K, status, stream);
}

#ifdef PLM_TEST_GIVE_UP
extern "C" int plm_test_give_up(int how, cudaStream_t stream) {
    return plm_status_of(cudaMemcpyToSymbolAsync(plm_give_up_switch, &how, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
}
#endif
