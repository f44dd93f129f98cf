// The experts' products of a routed feed-forward for few rows an expert (decode steps, short prompts), bfloat16: tiles of 16
// sorted rows of one expert each (routed.cu, moe_align) times the expert's weights on mma.sync m16n8k16, fp32 sums.
//
// The weights are what these products move: every element is used once a tile.  One CTA an SM stays and streams its share
// through a ring in shared memory (9 stages of 16 KB or 5 of 32: some 150 KB an SM asked for ahead, across columns and tiles):
// a thread issues the tensor copies (32 or 64 rows x 128 of K), a warp copies the tile's own rows beside them, and eight warps
// with eight columns each stand at the other end.  The columns of all tiles are dealt out 32 at a time, so that the busiest SM
// has at most 32 columns more than its share; where an expert has several tiles, a stretch of its columns goes to them in
// turn, and all but the first find the weights in the second-level cache.
// Blocks that read their weights straight into registers (what ran before) had 47 .. 56 % of the memory's rate (4,096 x 5,376,
// 32 pairs over 16 experts: up 144 us, down 171 us; a full wave and a ragged one of 1,400 blocks, each with a start and an
// end); this: 96 and 103 us in a row of launches, 111 and 113 alone.  (With the tile's rows in registers, loaded a stage ahead, a stage lasted as long as that load:
// 170 us.)
// The sums' order is that of the kernel for other sizes (moe_gemm_mma_kernel): the same bits.
#include "tc_common.cuh"

using namespace plm_tc;

namespace {

constexpr int CONSUMERS = 8, THREADS = (CONSUMERS + 2) * 32;
constexpr int BM16 = 16, GN = 32, KS = 128;            // rows of a tile, columns dealt out at a time, K of a stage
constexpr uint32_t COPY = GN * KS * 2;                 // bytes of GN columns of a stage
constexpr uint32_t ROWS = BM16 * KS * 2;               // bytes of the tile's rows in a stage
constexpr int MAX_TILES = 512;
enum { GATE_UP = 0, DOWN = 1, UP = 2 };                // as plm_moe_gemm's modes

template <int MODE> struct Ring {
    static constexpr uint32_t WEIGHTS = (MODE == GATE_UP ? 4 : 2) * COPY, STAGE = WEIGHTS + ROWS;
    static constexpr int STAGES = (int)(200000 / STAGE);
    static constexpr size_t SMEM = (size_t)STAGES * STAGE + 1024 + STAGES * 16;
};

// A tile's expert, and where among the tiles its expert's begin and how many they are.
struct Tiles { const int* expert; const unsigned short *first, *run; };

// Which columns of which tile come at place j of the order: `n` neighbouring pieces of GN columns, at most two.
struct Unit { int tile, piece, n; };
__device__ __forceinline__ Unit unit_at(int j, int end, const Tiles& tiles, int pieces) {
    const int first = tiles.first[j / pieces], run = tiles.run[j / pieces];
    const int at = j - first * pieces, paired = pieces / 2 * 2 * run;
    Unit u;
    if (at < paired) {
        const int in = at % (2 * run);
        u.tile = first + in / 2;
        u.piece = at / (2 * run) * 2 + in % 2;
        u.n = in % 2 == 0 && j + 1 < end ? 2 : 1;
    } else {
        u.tile = first + at - paired;
        u.piece = pieces - 1;
        u.n = 1;
    }
    return u;
}

// Where a row's 16-byte pieces lie: turned so that eight lanes (two rows of four pieces) read eight different banks.
__device__ __forceinline__ int row_turn(int row) { return ((row & 1) << 2) | ((row >> 1) & 3); }

template <int MODE>
__global__ void __launch_bounds__(THREADS, 1)
moe_stream_kernel(const __grid_constant__ CUtensorMap map_1, const __grid_constant__ CUtensorMap map_2, const bf16* a, long lda, int top,
                  void* __restrict__ out_, long ldo, const int* tile_expert, const int* sorted, int max_tiles, int N, int K, int interleaved,
                  int* status) {
    constexpr int NACC = MODE == GATE_UP ? 2 : 1, STAGES = Ring<MODE>::STAGES;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ int expert[MAX_TILES];
    __shared__ unsigned short first_of[MAX_TILES], run_of[MAX_TILES];
    __shared__ int n_tiles_, s_abort;
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    const uint32_t full0 = base + STAGES * Ring<MODE>::STAGE, empty0 = full0 + 8 * STAGES;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        n_tiles_ = 0;
        s_abort = 0;
        for (int s = 0; s < STAGES; ++s) { mbar_init(full0 + 8 * s, 1 + 32); mbar_init(empty0 + 8 * s, CONSUMERS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_launch_dependents();
    pdl_wait();
    __syncthreads();
    for (int i = tid; i < max_tiles; i += THREADS) {
        const int e = tile_expert[i];
        expert[i] = e;
        if (e >= 0) atomicMax(&n_tiles_, i + 1);
    }
    __syncthreads();
    const int n_tiles = n_tiles_, pieces = N / GN, n_stages = (K + KS - 1) / KS;
    // (the tiles come in ascending order of their experts; found once: with all tokens at one expert, walking its tiles for every
    // unit took 1.9 ms for a product of 140 us)
    for (int i = tid; i < n_tiles; i += THREADS) {
        const int e = expert[i];
        int lo = 0, hi = i;                            // the first tile of e
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (expert[mid] < e) lo = mid + 1; else hi = mid;
        }
        const int first = lo;
        hi = n_tiles, lo = i + 1;                      // the first behind its last
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (expert[mid] <= e) lo = mid + 1; else hi = mid;
        }
        first_of[i] = (unsigned short)first, run_of[i] = (unsigned short)(lo - first);
    }
    __syncthreads();
    const Tiles tiles = {expert, first_of, run_of};
    const long total = (long)n_tiles * pieces;
    const int begin = (int)(total * blockIdx.x / gridDim.x), end = (int)(total * (blockIdx.x + 1) / gridDim.x);

    if (warp == CONSUMERS) {
        // ------------------------------------------------------------ tensor copies
        if (elect_one()) {
            int i = 0;                                 // stages issued
            for (int j = begin; j < end;) {
                const Unit u = unit_at(j, end, tiles, pieces);
                const int n0 = u.piece * GN, row0 = expert[u.tile] * NACC * N;
                j += u.n;
                for (int s = 0; s < n_stages; ++s, ++i) {
                    const uint32_t bar = full0 + 8 * (i % STAGES), dst = base + (i % STAGES) * Ring<MODE>::STAGE;
                    if (*(volatile int*)&s_abort || !mbar_wait(empty0 + 8 * (i % STAGES), ((i / STAGES) & 1) ^ 1, status, 41)) { s_abort = 1; break; }
                    mbar_expect_tx(bar, u.n * NACC * COPY);
                    const CUtensorMap* map = u.n == 2 ? &map_2 : &map_1;
                    tma_load_3d(dst, map, bar, row0 + (MODE == GATE_UP && interleaved ? (n0 >> 6) * 128 + (n0 & 63) : n0), s * (KS / 64));
                    if (MODE == GATE_UP)
                        tma_load_3d(dst + 2 * COPY, map, bar, row0 + (interleaved ? (n0 >> 6) * 128 + 64 + (n0 & 63) : N + n0), s * (KS / 64));
                }
                if (*(volatile int*)&s_abort) break;
            }
            if (*(volatile int*)&s_abort)              // let what is in flight land
                for (int s = max(0, i - STAGES); s < i; ++s) mbar_wait(full0 + 8 * (s % STAGES), (s / STAGES) & 1, nullptr, 0);
        }
    } else if (warp == CONSUMERS + 1) {
        // ------------------------------------------------------------ the tile's rows: eight 16-byte pieces a lane and stage
        const int row = lane >> 1, first = (lane & 1) * 8;
        int i = 0, tile = -1;
        long off = -1;
        bool ok = true;
        for (int j = begin; j < end && ok;) {
            const Unit u = unit_at(j, end, tiles, pieces);
            j += u.n;
            if (u.tile != tile) {
                tile = u.tile;
                const int entry = sorted[tile * BM16 + row];
                off = entry < 0 ? -1 : (MODE != DOWN ? (long)(entry / top) * lda : (long)(tile * BM16 + row) * lda);
            }
            for (int s = 0; s < n_stages; ++s, ++i) {
                if (*(volatile int*)&s_abort || !mbar_wait(empty0 + 8 * (i % STAGES), ((i / STAGES) & 1) ^ 1, status, 43)) { s_abort = 1; ok = false; break; }
                const uint32_t dst = base + (i % STAGES) * Ring<MODE>::STAGE + Ring<MODE>::WEIGHTS + row * (KS * 2);
#pragma unroll
                for (int x = 0; x < 8; ++x) {
                    const int chunk = first + x, k = s * KS + chunk * 8;
                    const bool in = off >= 0 && k < K;                   // (elsewhere zeros, nothing is read)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                                 ::"r"(dst + ((chunk ^ row_turn(row)) << 4)), "l"(in ? a + off + k : a), "r"(in ? 16 : 0) : "memory");
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full0 + 8 * (i % STAGES)) : "memory");
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        // ------------------------------------------------------------ products
        // A lane's weight row among the warp's eight: neighbouring groups of four lanes read rows four apart, which the copies'
        // swizzle puts into different banks.
        const int g = lane >> 2, c = lane & 3, half = warp >> 2, row = (warp & 3) * 8 + (g >> 1) + (g & 1) * 4;
        int i = 0;
        bool ok = true;
        for (int j = begin; j < end && ok;) {
            const Unit u = unit_at(j, end, tiles, pieces);
            j += u.n;
            const bool mine = half < u.n;
            float acc[NACC][4];
#pragma unroll
            for (int m = 0; m < NACC; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;
            for (int s = 0; s < n_stages; ++s, ++i) {
                if (!mbar_wait_warp(full0 + 8 * (i % STAGES), (i / STAGES) & 1, status, 42)) { ok = false; s_abort = 1; break; }
                if (mine) {
                    const uint8_t* stage = smem_raw + (base - raw) + (i % STAGES) * Ring<MODE>::STAGE;
                    const uint8_t* at = stage + (half * GN + row) * 128;             // [64 of K][columns of the unit][128 bytes]
                    const uint8_t* rows = stage + Ring<MODE>::WEIGHTS + g * (KS * 2);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int place = (q >> 1) * u.n * (GN * 128) + ((((q & 1) * 4 + c) ^ (row & 7)) << 4);
                        const uint4 lo = *reinterpret_cast<const uint4*>(rows + (((q * 4 + c) ^ row_turn(g)) << 4));
                        const uint4 hi = *reinterpret_cast<const uint4*>(rows + 8 * KS * 2 + (((q * 4 + c) ^ row_turn(g)) << 4));
#pragma unroll
                        for (int m = 0; m < NACC; ++m) {
                            const uint4 b = *reinterpret_cast<const uint4*>(at + m * 2 * COPY + place);
                            asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                                         : "+f"(acc[m][0]), "+f"(acc[m][1]), "+f"(acc[m][2]), "+f"(acc[m][3])
                                         : "r"(lo.x), "r"(hi.x), "r"(lo.y), "r"(hi.y), "r"(b.x), "r"(b.y));
                            asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                                         : "+f"(acc[m][0]), "+f"(acc[m][1]), "+f"(acc[m][2]), "+f"(acc[m][3])
                                         : "r"(lo.z), "r"(hi.z), "r"(lo.w), "r"(hi.w), "r"(b.z), "r"(b.w));
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty0 + 8 * (i % STAGES)) : "memory");
            }
            if (!ok || !mine) continue;
            // c0, c1: row g, lanes' weight rows 2 c and 2 c + 1 (columns c and c + 4 of the warp's eight); c2, c3: row g + 8
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int at = u.tile * BM16 + g + 8 * r;
                if (sorted[at] < 0) continue;
                const size_t o = (size_t)at * ldo + (u.piece + half) * GN + (warp & 3) * 8 + c;
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    const float z = acc[0][2 * r + y];
                    if (MODE == GATE_UP) {
                        const float gv = __bfloat162float(__float2bfloat16_rn(z)), uv = __bfloat162float(__float2bfloat16_rn(acc[NACC - 1][2 * r + y]));
                        reinterpret_cast<bf16*>(out_)[o + 4 * y] = __float2bfloat16_rn(gv / (1.0f + expf(-gv)) * uv);
                    } else if (MODE == UP) {
                        const float p = fmaxf(z, 0.f);
                        reinterpret_cast<bf16*>(out_)[o + 4 * y] = __float2bfloat16_rn(p * p);
                    } else {
                        reinterpret_cast<float*>(out_)[o + 4 * y] = z;
                    }
                }
            }
        }
    }
}

template <int MODE>
int launch(const CUtensorMap& map_1, const CUtensorMap& map_2, const void* a, long lda, int top, void* out, long ldo, const int* tile_expert,
           const int* sorted, int max_tiles, int N, int K, int interleaved, int* status, cudaStream_t stream) {
    static std::atomic<unsigned long long> devices{0};
    const cudaError_t configured = plm_allow_smem(moe_stream_kernel<MODE>, Ring<MODE>::SMEM, devices);
    if (configured != cudaSuccess) return (int)configured;
    const long most = (long)max_tiles * (N / GN);
    return plm_status_of(launch_pdl(moe_stream_kernel<MODE>, dim3((unsigned)(most < PLM_SM_COUNT ? most : PLM_SM_COUNT)), dim3(THREADS),
                                    Ring<MODE>::SMEM, stream, map_1, map_2, (const bf16*)a, lda, top, out, ldo, tile_expert, sorted, max_tiles,
                                    N, K, interleaved, status));
}

}  // namespace

// plm_moe_gemm's products (same arguments; `n_experts`: how many experts' weights w holds) for bfloat16 and tiles of 16 rows,
// N a multiple of 32 and K of 64.  `status`: a device int that stays 0 unless a bounded wait ran out.
extern "C" int plm_moe_stream(const void* a, long lda, int top, const void* w, int n_experts, void* out, long ldo, int mode,
                              const int* tile_expert, const int* sorted, int max_tiles, int N, int K, int interleaved, int* status,
                              cudaStream_t stream) {
    if (max_tiles <= 0) return PLM_OK;
    if (N <= 0 || K <= 0 || top <= 0 || n_experts <= 0 || mode < 0 || mode > 2 || (interleaved && (mode != 0 || N % 64))) return PLM_ERR_SHAPE;
    if (max_tiles > MAX_TILES || N % GN || K % 64) return PLM_ERR_UNSUPPORTED;
    if (lda % 8 || (((uintptr_t)a | (uintptr_t)w) & 15) || ((uintptr_t)out & 3)) return PLM_ERR_ALIGN;
    CUtensorMap one, two;                  // pieces of 32 columns alone and in pairs
    const long w_rows = (long)n_experts * (mode == GATE_UP ? 2 : 1) * N;
    int rc = make_map(&one, w, w_rows, K, K, GN, KS / 64);
    if (rc == PLM_OK) rc = make_map(&two, w, w_rows, K, K, 2 * GN, KS / 64);
    if (rc != PLM_OK) return rc;
    if (mode == GATE_UP) return launch<GATE_UP>(one, two, a, lda, top, out, ldo, tile_expert, sorted, max_tiles, N, K, interleaved, status, stream);
    if (mode == DOWN) return launch<DOWN>(one, two, a, lda, top, out, ldo, tile_expert, sorted, max_tiles, N, K, interleaved, status, stream);
    return launch<UP>(one, two, a, lda, top, out, ldo, tile_expert, sorted, max_tiles, N, K, interleaved, status, stream);
}
