// Grouped matrix products of a mixture of experts on the fifth-generation tensor cores (tcgen05), bf16.
//
// The rows of X [P, K] are the steps' (token, expert) pairs sorted by expert, W holds the experts' matrices one below the
// other (N rows of K each), and every row is multiplied by its expert's matrix:
//   plain   C[p, :] = X[p, :] W_e^T                                      (kExpPlain; kExpRelu2: relu(T(.))^2)
//   gated   C[p, :] = f(T(X Wg_e^T), T(X Wu_e^T)),  W_e = [Wg_e; Wu_e]   (kExpSwiglu, kExpClamped)
//
// What bounds it.  Many rows per expert: the power limit.  8 experts of 512 pairs, K 4,096, 9,472 gated weight rows run at 1,385
// TFLOP/s while the clock falls from 1.6 to 1.2 GHz (a cuBLAS product in a row on this machine: 1,383), so what is left to gain is
// work not done.  Two SMs as a pair (cta_group::2, 256 x 256 a tile) take 32 KB a stage from the L2 each where one SM takes 48 for
// the same products (1,320).  Few rows: the weights, read once from memory at 4.1 to 5.5 TB/s with up to 192 KB of TMA copies in
// flight per SM.  2,048 tokens, two of 8 experts of 151 MB: 354 + 284 us with tiles of 128 pairs by 256 weight rows on one SM and
// segments padded to 128 pairs, now 322 + 190 (128 tokens: 180 + 157, now 205 + 100; 600: 205 + 131, now 182 + 107).
//
// The weights are the M operand and the pairs the N operand: an expert's rows are cut into tiles of at most 256 pairs, all
// nearly as large, and N is rounded up to 32 (16 on one SM) and no further, so ragged segments cost no padding and
// need no alignment.  A tile's accumulator has a weight row per lane and a pair per column; the epilogue turns 32 pairs by
// 128 weight rows at a time through shared memory and writes whole lines.  A gated tile's 128 lanes are 64 gate rows over
// the 64 matching up rows, which meet there.
//
// One persistent cluster of CTAS blocks per pair of SMs (per SM with CTAS = 1) walks the units (expert, 128 * CTAS weight
// rows, tile of pairs), tiles of pairs fastest, so that the clusters that run side by side share the weight rows they read.
// Roles, by warp:
//   warp 0   producer: its block's 128 weight rows and its share (N / CTAS rows) of the pairs of every block of 64 of K into
//            a ring of stages by TMA (128-byte swizzle).  Both blocks' copies are counted on the first block's "full" mbarrier;
//   warp 1   tensor memory (two accumulators of 256 columns); in the first block one thread issues the products and the
//            commits, which arrive in both blocks: on "empty" when a stage has been read, on "ready" when a tile is done;
//   warps 2-5 epilogue: tile i drains accumulator i % 2 while tile i + 1 fills the other.
// Every wait is bounded by a cycle count; one that runs out records error 5 and the block carries on to its end.
#include "sm100.cuh"
#include "tensor_map.cuh"

namespace cvb {

constexpr int kExpThreads = 192;
constexpr int kExpRows = 128;                 // weight rows of a block (lanes of its accumulator)
constexpr int kExpPairs = 256;                // most pairs of a tile (columns of an accumulator)
constexpr int kExpBK = 64;                    // one 128-byte swizzle span of bf16
constexpr int kExpPitch = 320;                // bytes between pairs in the epilogue's shared memory: 128 weight rows and 64 bytes
constexpr int kExpTable = 1024;               // experts whose segment table is kept in shared memory

enum ExpertEpilogue { kExpPlain = 0, kExpSwiglu = 1, kExpRelu2 = 3, kExpClamped = 4 };
constexpr bool expert_gated(int e) { return e == kExpSwiglu || e == kExpClamped; }

struct ExpertParams {
    __nv_bfloat16* out;       // [P, n_out]
    const int* start;         // [E + 1] first sorted row of each expert; [E]: all rows
    const int* tiles;         // [E + 1] tiles of pairs before each expert
    int K, N, n_out, E;       // N: weight rows of one expert; n_out: N, or N / 2 when gated
    int feature_tiles;
    float limit, alpha;       // kExpClamped
    int* err;
};

template <int CTAS> struct ExpertSmem {
    static constexpr int kABytes = kExpRows * kExpBK * 2;
    static constexpr int kBBytes = kExpPairs / CTAS * kExpBK * 2;
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kStages = CTAS == 2 ? 6 : 4;
    static constexpr int kBufBytes = 32 * kExpPitch;
    static constexpr size_t kBytes = 1024 + static_cast<size_t>(kStages) * kStageBytes + 2 * kBufBytes + (2 * kStages + 4) * 8 + 16 + 2 * (kExpTable + 1) * 4;
};

// ---- instructions of a pair of blocks --------------------------------------------------------------------------------------

// the shared-memory address `local` as block `rank` of the cluster has it
__device__ __forceinline__ uint32_t cluster_addr(const void* local, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"(smem_u32(local)), "r"(rank));
    return a;
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
// one box into this block's shared memory; of a pair of blocks, counted on a barrier of either
__device__ __forceinline__ void tma_load_3d(void* smem, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n"
                 ::"r"(smem_u32(smem)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void* smem, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n"
                 ::"r"(smem_u32(smem)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(void* smem, const CUtensorMap* map, uint32_t bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
                 ::"r"(smem_u32(smem)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                 ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// one arrival on the barrier at this address in both blocks
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
                 ::"r"(smem_u32(bar)), "h"(static_cast<uint16_t>(3)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// bounded wait for what either block of the pair did before it arrived
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n.reg .pred P1;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P1, [%1], %2;\nselp.b32 %0, 1, 0, P1;\n}\n"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void mbar_wait_cluster(uint64_t* bar, uint32_t parity, int* err) {
    if (mbar_try_wait_cluster(bar, parity)) return;
    const long long t0 = clock64();
    while (!mbar_try_wait_cluster(bar, parity)) {
        if (clock64() - t0 > 40000000LL) { atomicExch(err, 5); return; }
    }
}

// ---- the walk over units ---------------------------------------------------------------------------------------------------

struct ExpertUnit { int expert, feature, row0, rows; };

// Unit u, given the expert of an earlier one (units are asked for in rising order); false behind the last.
__device__ __forceinline__ bool expert_unit(int u, const int* start, const int* tiles, const ExpertParams& p, int& e, ExpertUnit& out) {
    const int ft = p.feature_tiles;
    while (e < p.E && u >= ft * tiles[e + 1]) ++e;
    if (e >= p.E) return false;
    const int first = tiles[e], n_tiles = tiles[e + 1] - first, r = u - ft * first, f = r / n_tiles, t = r - f * n_tiles;
    const int n = start[e + 1] - start[e];
    const int per = ((n + n_tiles - 1) / n_tiles + 15) & ~15;      // at most the tile's limit, which is a multiple of 16, so no tile is empty
    out.expert = e;
    out.feature = f;
    out.row0 = start[e] + t * per;
    out.rows = min(per, n - t * per);
    return true;
}

template <int EPI>
__device__ __forceinline__ float expert_gated_value(float g, float u, float limit, float alpha) {
    if constexpr (EPI == kExpClamped) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
        return __fdividef(g, 1.f + __expf(-alpha * g)) * (u + 1.f);
    } else {
        return rnd<__nv_bfloat16>(__fdividef(g, 1.f + __expf(-g))) * u;
    }
}

template <int CTAS, int EPI>
__global__ void __launch_bounds__(kExpThreads)
gemm_experts_kernel(const __grid_constant__ CUtensorMap map_x32, const __grid_constant__ CUtensorMap map_x64, const __grid_constant__ CUtensorMap map_x128,
                    const __grid_constant__ CUtensorMap map_w, const ExpertParams p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    using L = ExpertSmem<CTAS>;
    constexpr bool GATED = expert_gated(EPI);
    constexpr int STAGES = L::kStages;
    constexpr int OUT_COLS = GATED ? kExpRows / 2 : kExpRows;      // output columns of a block
    pdl_trigger();
    const uint32_t raw_addr = smem_u32(smem_raw);
    unsigned char* stages = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
    unsigned char* bufs = stages + static_cast<size_t>(STAGES) * L::kStageBytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(bufs + 2 * L::kBufBytes);     // used in the first block of a cluster
    uint64_t* empty = full + STAGES;
    uint64_t* acc_ready = empty + STAGES;              // [2]
    uint64_t* acc_free = acc_ready + 2;                // [2]  used in the first block: four warps of each block
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 2);
    int* table = reinterpret_cast<int*>(tmem_slot + 4);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = CTAS == 2 ? static_cast<int>(cluster_rank()) : 0;
    const int first_unit = blockIdx.x / CTAS, unit_step = gridDim.x / CTAS;
    const int num_kb = (p.K + kExpBK - 1) / kExpBK;

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) { mbar_init(full + i, 1); mbar_init(empty + i, 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(acc_ready + i, 1); mbar_init(acc_free + i, 4 * CTAS); }
        mbar_fence_init();
    }
    if (warp == 1) {
        if constexpr (CTAS == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(2 * kExpPairs));
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::);
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(2 * kExpPairs));
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
        }
    }
    pdl_wait();                                        // the pairs and their table come from the kernels before this one
    const int* start = p.start;
    const int* tiles = p.tiles;
    if (p.E <= kExpTable) {
        for (int i = threadIdx.x; i <= p.E; i += kExpThreads) {
            table[i] = p.start[i];
            table[p.E + 1 + i] = p.tiles[i];
        }
        start = table;
        tiles = table + p.E + 1;
    }
    tc_before();
    __syncthreads();
    if constexpr (CTAS == 2) cluster_sync();           // both blocks' barriers are there
    tc_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {                               // ---- producer ----
            int it = 0, e = 0;
            ExpertUnit t;
            for (int u = first_unit; expert_unit(u, start, tiles, p, e, t); u += unit_step) {
                const int share = CTAS == 2 ? ((t.rows + 31) / 32) * 16 : (t.rows + 15) / 16 * 16;     // pairs this block brings
                const int box_rows = share <= 32 ? 32 : (share <= 64 ? 64 : 128);
                const CUtensorMap* map_x = share <= 32 ? &map_x32 : (share <= 64 ? &map_x64 : &map_x128);
                const bool two = CTAS == 1 && share > 128;
                const uint32_t bytes = L::kABytes + (two ? 2 : 1) * box_rows * (kExpBK * 2);
                const int f0 = (t.feature * CTAS + rank) * OUT_COLS, x0 = t.row0 + rank * share, plane = GATED ? 2 * t.expert : t.expert;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % STAGES;
                    unsigned char* a_dst = stages + static_cast<size_t>(s) * L::kStageBytes;
                    unsigned char* b_dst = a_dst + L::kABytes;
                    if constexpr (CTAS == 2) {
                        if (it >= STAGES) mbar_wait_cluster(empty + s, ((it / STAGES) - 1) & 1, p.err);
                        const uint32_t bar = cluster_addr(full + s, 0);
                        if (rank == 0) mbar_expect_tx(full + s, 2 * bytes);
                        tma_load_3d_pair(a_dst, &map_w, bar, kb * kExpBK, f0, plane);
                        tma_load_2d_pair(b_dst, map_x, bar, kb * kExpBK, x0);
                    } else {
                        if (it >= STAGES) mbar_wait(empty + s, ((it / STAGES) - 1) & 1, p.err);
                        mbar_expect_tx(full + s, bytes);
                        tma_load_3d(a_dst, &map_w, full + s, kb * kExpBK, f0, plane);
                        tma_load_2d(b_dst, map_x, full + s, kb * kExpBK, x0);
                        if (two) tma_load_2d(b_dst + 128 * kExpBK * 2, map_x, full + s, kb * kExpBK, x0 + 128);
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {                  // ---- tensor-core issue, for both blocks ----
            int it = 0, i = 0, e = 0;
            ExpertUnit t;
            for (int u = first_unit; expert_unit(u, start, tiles, p, e, t); u += unit_step, ++i) {
                const int buf = i & 1, use = i >> 1;
                if (use > 0) {                         // the epilogue of the tile before last has drained this accumulator
                    if constexpr (CTAS == 2) mbar_wait_cluster(acc_free + buf, (use - 1) & 1, p.err);
                    else mbar_wait(acc_free + buf, (use - 1) & 1, p.err);
                    tc_after();
                }
                const int n = CTAS == 2 ? (t.rows + 31) / 32 * 32 : (t.rows + 15) / 16 * 16;
                const uint32_t idesc = idesc_bf16(kExpRows * CTAS, n, false);
                const uint32_t tmem_d = tmem_base + buf * kExpPairs;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % STAGES;
                    if constexpr (CTAS == 2) mbar_wait_cluster(full + s, (it / STAGES) & 1, p.err);
                    else mbar_wait(full + s, (it / STAGES) & 1, p.err);
                    tc_after();
                    const uint32_t a_addr = smem_u32(stages + static_cast<size_t>(s) * L::kStageBytes);
                    const uint32_t b_addr = a_addr + L::kABytes;
#pragma unroll
                    for (int k = 0; k < kExpBK / 16; ++k) {
                        const uint64_t da = desc_sw128(a_addr + k * 32, 16, 1024), db = desc_sw128(b_addr + k * 32, 16, 1024);
                        if constexpr (CTAS == 2) umma_pair(tmem_d, da, db, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                        else umma(tmem_d, da, db, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    }
                    if constexpr (CTAS == 2) tc_commit_pair(empty + s); else tc_commit(empty + s);
                }
                if constexpr (CTAS == 2) tc_commit_pair(acc_ready + buf); else tc_commit(acc_ready + buf);
            }
        }
    } else {                                           // ---- epilogue: warps 2..5 own lanes 32 * (warp % 4) .. +31 ----
        const int quarter = warp & 3, tid = threadIdx.x - 64;
        int i = 0, e = 0, chunk = 0;
        ExpertUnit t;
        for (int u = first_unit; expert_unit(u, start, tiles, p, e, t); u += unit_step, ++i) {
            const int buf = i & 1, use = i >> 1;
            const uint32_t tmem_d = tmem_base + buf * kExpPairs + (static_cast<uint32_t>(quarter * 32) << 16);
            const int n0 = (t.feature * CTAS + rank) * OUT_COLS;   // first output column of this block
            if constexpr (CTAS == 2) mbar_wait_cluster(acc_ready + buf, use & 1, p.err);
            else mbar_wait(acc_ready + buf, use & 1, p.err);
            tc_after();
#pragma unroll 1
            for (int c0 = 0; c0 < t.rows; c0 += 32, ++chunk) {
                unsigned char* st = bufs + (chunk & 1) * L::kBufBytes;
                uint32_t v[32];
                tm_load32(tmem_d + c0, v);
                tm_wait_ld();
                if (c0 + 32 >= t.rows) {               // the accumulator has been read
                    tc_before();
                    __syncwarp();
                    if (lane == 0) {
                        if constexpr (CTAS == 2) mbar_arrive_cluster(cluster_addr(acc_free + buf, 0)); else mbar_arrive(acc_free + buf);
                    }
                }
                // pair j of the chunk, weight row `quarter * 32 + lane`: a warp's 32 values of a pair lie side by side
                __nv_bfloat16* mine = reinterpret_cast<__nv_bfloat16*>(st) + quarter * 32 + lane;
#pragma unroll
                for (int j = 0; j < 32; ++j) mine[j * (kExpPitch / 2)] = __float2bfloat16_rn(__uint_as_float(v[j]));
                asm volatile("bar.sync 1, 128;\n" ::: "memory");   // also: everyone is done with the other buffer
                constexpr int PER_ROW = OUT_COLS / 8;              // 16-byte pieces of a pair's output
#pragma unroll
                for (int q = tid; q < 32 * PER_ROW; q += 128) {
                    const int j = q / PER_ROW, c = q - j * PER_ROW, col = n0 + c * 8;
                    if (c0 + j < t.rows && col < p.n_out) {
                        uint4 a = *reinterpret_cast<const uint4*>(st + j * kExpPitch + c * 16);
                        __nv_bfloat162* ha = reinterpret_cast<__nv_bfloat162*>(&a);
                        if constexpr (GATED) {
                            const uint4 b = *reinterpret_cast<const uint4*>(st + j * kExpPitch + 128 + c * 16);
                            const __nv_bfloat162* hb = reinterpret_cast<const __nv_bfloat162*>(&b);
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const float2 g = __bfloat1622float2(ha[k]), w = __bfloat1622float2(hb[k]);
                                ha[k] = __floats2bfloat162_rn(expert_gated_value<EPI>(g.x, w.x, p.limit, p.alpha),
                                                              expert_gated_value<EPI>(g.y, w.y, p.limit, p.alpha));
                            }
                        }
                        if constexpr (EPI == kExpRelu2) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                float2 g = __bfloat1622float2(ha[k]);
                                g.x = fmaxf(g.x, 0.f); g.y = fmaxf(g.y, 0.f);
                                ha[k] = __floats2bfloat162_rn(g.x * g.x, g.y * g.y);
                            }
                        }
                        *reinterpret_cast<uint4*>(p.out + static_cast<int64_t>(t.row0 + c0 + j) * p.n_out + col) = a;
                    }
                }
            }
        }
    }
    tc_before();
    __syncthreads();
    if constexpr (CTAS == 2) cluster_sync();           // neither block leaves while the other may still reach into it
    if (warp == 1) {
        tc_after();
        if constexpr (CTAS == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(2 * kExpPairs));
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(2 * kExpPairs));
    }
}

// ---- host side --------------------------------------------------------------------------------------------------------------

template <int CTAS, int EPI>
static int launch_experts(const CUtensorMap (&mx)[3], const CUtensorMap& mw, ExpertParams p, int most_tiles, cudaStream_t stream) {
    using L = ExpertSmem<CTAS>;
    static bool set = false;
    if (!set) {
        cudaError_t e = cudaFuncSetAttribute(gemm_experts_kernel<CTAS, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(L::kBytes));
        if (e != cudaSuccess) return static_cast<int>(e);
        set = true;
    }
    static int sms = 0;
    if (sms == 0) {
        int dev = 0, n = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 1) n = 148;
        sms = n;
    }
    const int cols = CTAS * (expert_gated(EPI) ? kExpRows / 2 : kExpRows);
    p.feature_tiles = (p.n_out + cols - 1) / cols;
    const int64_t units = static_cast<int64_t>(p.feature_tiles) * most_tiles;
    if (units > 2147483647LL) return CVB_E_SIZE;
    const int64_t clusters = units < sms / CTAS ? units : sms / CTAS;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(clusters * CTAS));
    cfg.blockDim = dim3(kExpThreads);
    cfg.dynamicSmemBytes = L::kBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (CTAS == 2) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 2;
        attr[n].val.clusterDim.y = 1;
        attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (pdl_enabled() && cudaStreamIsCapturing(stream, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    cudaLaunchKernelEx(&cfg, gemm_experts_kernel<CTAS, EPI>, mx[0], mx[1], mx[2], mw, p);
    return launch_status();
}

}  // namespace cvb

using namespace cvb;

// X [P, K]: the pairs' rows sorted by expert; segments [2 (E + 1)]: first row of every expert, then tiles of pairs before every
// expert (sort_pairs in moe.cu, which was given the same `tile_pairs`); W [E * N, K].  mode 0: C [P, N];  mode 1: C [P, N / 2] with
// silu;  mode 3: relu^2;  mode 4: like 1 with the clamped activation.  pair_ctas: blocks that share a tile, 1 or 2.
extern "C" int cvb_gemm_experts_bf16(void* out, const void* x, const void* w, const int* segments, int P, int N, int E, int K, int mode,
                                     int tile_pairs, int pair_ctas, float limit, float alpha, int* err_flag, cudaStream_t stream) {
    if (P == 0) return CVB_OK;
    if (P < 0 || N <= 0 || K <= 0 || E <= 0 || segments == nullptr) return CVB_E_SIZE;
    if (K % 8) return CVB_E_ALIGN;
    auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    if (!al(out) || !al(x) || !al(w)) return CVB_E_ALIGN;
    if (mode != 0 && mode != 1 && mode != 3 && mode != 4) return CVB_E_SHAPE;
    if (tile_pairs < 32 || tile_pairs > kExpPairs || tile_pairs % 32 || (pair_ctas != 1 && pair_ctas != 2)) return CVB_E_SHAPE;
    const bool gated = mode == 1 || mode == 4;
    if (gated && (N % 2)) return CVB_E_SHAPE;
    if (static_cast<int64_t>(E) * N > 2147483647LL) return CVB_E_SIZE;
    ExpertParams p{};
    p.out = (__nv_bfloat16*)out; p.start = segments; p.tiles = segments + E + 1;
    p.K = K; p.N = N; p.n_out = gated ? N / 2 : N; p.E = E; p.limit = limit; p.alpha = alpha; p.err = err_flag;
    if (p.n_out % 8) return CVB_E_ALIGN;               // 16-byte stores of output rows
    // One copy of a stage's weight rows and one of its pairs: 128 weight rows (64 gate and the 64 matching up rows as two planes),
    // and the smallest box that holds a block's share of the pairs.  Boxes of 32 pairs and of 64 weight rows took 538 ns a
    // stage of 2 x 32 KB where these take 464 (8 experts of 512 pairs, K 4,096): a copy costs more the smaller its box is.
    CUtensorMap mx[3], mw;
    for (int i = 0; i < 3; ++i) {
        const int rc = cached_bf16_map(&mx[i], x, P, K, kExpBK, 32 << i);
        if (rc != CVB_OK) return rc;
    }
    const int rc = gated ? cached_bf16_map(&mw, w, p.n_out, K, kExpBK, 64, 2LL * E, 2) : cached_bf16_map(&mw, w, p.n_out, K, kExpBK, 128, E, 1);
    if (rc != CVB_OK) return rc;
    const int most = P / tile_pairs + (P < E ? P : E);
#define CALL(EPI) return pair_ctas == 2 ? launch_experts<2, EPI>(mx, mw, p, most, stream) : launch_experts<1, EPI>(mx, mw, p, most, stream)
    if (mode == 1) CALL(kExpSwiglu);
    if (mode == 4) CALL(kExpClamped);
    if (mode == 3) CALL(kExpRelu2);
    CALL(kExpPlain);
#undef CALL
}
