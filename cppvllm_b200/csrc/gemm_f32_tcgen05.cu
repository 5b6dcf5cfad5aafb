// Matrix product of the 32-bit path on the fifth-generation tensor cores (tcgen05):
//   C[M, N] = A[M, K] * W[N, K]^T,  all float32, with the error of a product in float32.
//
// The tensor cores multiply 16-bit operands far faster than the float units add up 32-bit ones, so every element is cut into
// three bf16 parts, a = a0 + a1 + a2: a0 is a rounded to nearest, a1 what is left rounded to nearest, a2 the rest, which has at most
// eight bits left.  The cuts are exact: |a1| <= 2^-8 |a|, |a2| <= 2^-17 |a|, and nothing of the 24 bits is lost.  Of the nine products of parts,
// the six of weight 2^0, 2^-8 and 2^-16 are taken; what is left out (a1 w2, a2 w1, a2 w2) is at most 2^-24 (1 + 2^-9) of |a w|, of either sign, no
// more than the rounding of a float32 product.  (Parts cut off instead of rounded leave up to 2^-21 out, always towards zero:
// operands just above a bf16 came out 4.7e-7 too small.)  Products of parts are exact in the float accumulators' inputs.  The tensor
// core's accumulation truncates where a float add rounds, so a chain in tensor memory is kept short: after every 128 of K the partial sums
// (those of weight 2^0 apart from the smaller ones) are read back and added, rounded to nearest, to sums in registers.  Error against
// float64, 17 to 449 rows, K 128 to 8,192: 0.7e-7 to 1.5e-7 for operands of both signs (the library's float32 product 2.0e-7 to 8.1e-7), 0.8e-7 to
// 1.5e-7 for operands of one sign (1.4e-7 to 6.0e-7), where truncation makes nearly all of it.
//
// A block makes 128 columns of C (rows of W: the M operand) for up to 128 rows of A (the N operand, rounded up to 32):
//   warps 0-7   fetch the next 64 of K of both operands (16 bytes a thread), cut them and lay the parts into shared memory as
//               128-byte swizzled tiles, one tile per part, 2 or 3 stages;
//   warp 8      also issues the products, one stage ahead of its sums.  Up to 64 rows of A, the parts of A lie one below the other, so that w0 meets
//               [a0 a1 a2], w1 [a0 a1] and w2 [a0] in three products that read W's parts once each, and equal weights share
//               columns;  more rows: one product per pair of parts, w0 a0 in one accumulator, the five smaller in another;
//   warps 8-15  add the partial sums of the stage before (accumulators alternate) and store C.
// With few tiles the blocks of a cluster share a tile's K and add their sums up through distributed shared memory.
//
// What bounds it: no unit alone.  At 2,048 rows by 4,096 x 4,096 the tensor pipe is active for 54 % of the cycles, shared memory (a product of
// parts of 128 x 128 x 16 reads 8 KB in the 64 cycles it takes, and the parts have to be written) for 61, the issue slots, mostly the cuts', for
// 45, and the cutting warps wait for their rows from the L2 or memory (W is read again by every 128 rows of A: 327 MB where 101 are
// needed).  449 rows by 4,096 x 1,024: 86 us as a float32
// library product, 33 with parts cut off, now 28 (134 TFLOP/s of float32 work); by 1,024 x 2,048 57, 21, now 18; 2,048 rows by 4,096 x 1,024 330,
// 128, now 108 (159 TFLOP/s).
// Every wait is bounded by a cycle count; one that runs out records error 5 and the block carries on to its end.  The kernel may start while
// the ones before it run, for as long as those take, so the threads ask for W alone and pass griddepcontrol.wait before they wait
// for anything else.
#include "sm100.cuh"

namespace cvb {

constexpr int kSplitThreads = 16 * 32;
constexpr int kSplitRows = 128;               // rows of W a block
constexpr int kSplitBK = 64;                  // of K a stage: one 128-byte swizzle span of bf16
constexpr int kSplitFlush = 2;                // stages whose products add up in tensor memory
constexpr int kSplitStack = 64;               // rows of A up to which its parts are stacked
constexpr int kSplitABytes = kSplitRows * 128;

struct SplitParams {
    float* out;               // [M, N]
    const float* a;           // [M, K]
    const float* w;           // [N, K]
    int M, N, K;
    int* err;
};

// Two floats at once
__device__ __forceinline__ uint64_t pack2(float a, float b) { return static_cast<uint64_t>(__float_as_uint(a)) | (static_cast<uint64_t>(__float_as_uint(b)) << 32); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) { uint64_t d; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
// Two bf16 side by side: rounded to nearest, or the upper halves, which are all of a number of up to eight bits
__device__ __forceinline__ uint32_t nearest2(uint64_t v) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(__uint_as_float(static_cast<uint32_t>(v >> 32))), "f"(__uint_as_float(static_cast<uint32_t>(v))));
    return d;
}
__device__ __forceinline__ uint32_t upper_halves(uint64_t v) { return __byte_perm(static_cast<uint32_t>(v), static_cast<uint32_t>(v >> 32), 0x7632); }
// What two bf16 leave of two floats, exactly
__device__ __forceinline__ uint64_t rest2(uint64_t v, uint32_t h) { return sub2(v, static_cast<uint64_t>(h << 16) | (static_cast<uint64_t>(h & 0xFFFF0000u) << 32)); }

// Four consecutive elements into the three tiles of parts: 8 bytes each, `plane` bytes apart.
__device__ __forceinline__ void store_parts(unsigned char* at, uint32_t plane, float4 f) {
    uint64_t x = pack2(f.x, f.y), y = pack2(f.z, f.w);
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const uint32_t hx = nearest2(x), hy = nearest2(y);
        *reinterpret_cast<uint2*>(at + p * plane) = make_uint2(hx, hy);
        x = rest2(x, hx);
        y = rest2(y, hy);
    }
    *reinterpret_cast<uint2*>(at + 2 * plane) = make_uint2(upper_halves(x), upper_halves(y));
}

// A result that is not finite is computed again: an infinity, or a number that rounds to one, has no finite parts.
__device__ __forceinline__ void split_store(const SplitParams& p, int m, int n, float v) {
    if (!isfinite(v)) {
        const float* x = p.a + static_cast<int64_t>(m) * p.K;
        const float* y = p.w + static_cast<int64_t>(n) * p.K;
        v = 0.f;
#pragma unroll 1
        for (int k = 0; k < p.K; ++k) v = fmaf(x[k], y[k], v);
    }
    p.out[static_cast<int64_t>(m) * p.N + n] = v;
}

template <int NT>
__global__ void __launch_bounds__(kSplitThreads, 1)
gemm_f32_split_kernel(const SplitParams p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    pdl_trigger();
    const uint32_t raw_addr = smem_u32(smem_raw);
    unsigned char* base = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
    constexpr uint32_t b_plane = NT * 128, stage_bytes = 3 * (kSplitABytes + b_plane);
    constexpr bool stacked = NT <= kSplitStack;
    constexpr int STAGES = stacked ? 3 : 2;
    unsigned char* stage0 = base;
    uint64_t* full = reinterpret_cast<uint64_t*>(base + static_cast<size_t>(STAGES) * stage_bytes);   // [3]
    uint64_t* empty = full + 3;                        // [3]
    uint64_t* acc_ready = empty + 3;                   // [2]
    uint64_t* acc_free = acc_ready + 2;                // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 2);

    const int warp = same_in_warp(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int w0 = blockIdx.x * kSplitRows, m0 = blockIdx.y * NT;
    // the block's share of K, in stages from kb0; a cluster's blocks share a tile of C (grid.z), none without a stage
    const int all_kb = (p.K + kSplitBK - 1) / kSplitBK;
    const int kb0 = static_cast<int>(static_cast<int64_t>(all_kb) * blockIdx.z / gridDim.z);
    const int num_kb = static_cast<int>(static_cast<int64_t>(all_kb) * (blockIdx.z + 1) / gridDim.z) - kb0;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 3; ++i) { mbar_init(full + i, 8); mbar_init(empty + i, 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(acc_ready + i, 1); mbar_init(acc_free + i, 8); }
        mbar_fence_init();
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp < 8) {                                    // ---- cuts: 16 threads a row of 64, 16 rows at a time ----
        const int c = threadIdx.x, r = c >> 4, q = c & 15, k0 = kb0 * kSplitBK + q * 4;
        constexpr int A_ITEMS = NT / 16;
        // Byte offsets of the thread's rows; rows behind the last repeat it (their results are not stored).
        uint32_t w_at[8], a_at[A_ITEMS];
#pragma unroll
        for (int i = 0; i < 8; ++i) w_at[i] = (static_cast<uint32_t>(min(w0 + r + 16 * i, p.N - 1)) * p.K + k0) * 4;
#pragma unroll
        for (int i = 0; i < A_ITEMS; ++i) a_at[i] = (static_cast<uint32_t>(min(m0 + r + 16 * i, p.M - 1)) * p.K + k0) * 4;
        float4 wv[8], av[A_ITEMS];
        // a row of 64 is fetched again as soon as it has been cut, so every fetch has a whole stage to arrive
        auto load = [&](const float* base, uint32_t at, int kb) {
            return kb < num_kb && kb * kSplitBK + k0 < p.K ? *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(base) + (at + kb * (kSplitBK * 4u)))
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        // row r + 16 i keeps its place modulo 8, and with it the order of its 16-byte pieces
        const uint32_t place = r * 128 + (((q >> 1) ^ (r & 7)) << 4) + (q & 1) * 8;
#pragma unroll
        for (int i = 0; i < 8; ++i) wv[i] = load(p.w, w_at[i], 0);
        pdl_wait();                                    // the rows of A come from the kernel before this one
#pragma unroll
        for (int i = 0; i < A_ITEMS; ++i) av[i] = load(p.a, a_at[i], 0);
        for (int kb = 0, s = 0, round = 0; kb < num_kb; ++kb) {
            if (round > 0) mbar_wait(empty + s, (round - 1) & 1, p.err);
            unsigned char* at = stage0 + static_cast<size_t>(s) * stage_bytes + place;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                store_parts(at + i * 16 * 128, kSplitABytes, wv[i]);
                wv[i] = load(p.w, w_at[i], kb + 1);
            }
            at += 3 * kSplitABytes;
#pragma unroll
            for (int i = 0; i < A_ITEMS; ++i) {
                store_parts(at + i * 16 * 128, b_plane, av[i]);
                av[i] = load(p.a, a_at[i], kb + 1);
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(full + s);
            if (++s == STAGES) { s = 0; ++round; }
        }
    } else {                                           // ---- sums: two warps per 32 lanes, half of the columns each ----
        pdl_wait();                                    // before the first bounded wait: its limit is not for the time of the kernels before this one
        const int quarter = warp & 3, half = (warp - 8) >> 2;
        constexpr int COLS = NT / 2;
        // the products of stage kb: warp 8 walks them with values that are the same in all lanes, one lane issues
        constexpr uint32_t id1 = idesc_bf16(128, NT, false), id2 = idesc_bf16(128, 2 * NT, false), id3 = idesc_bf16(128, 3 * NT, false);
        const uint64_t desc = desc_sw128(smem_u32(stage0), 16, 1024);
        const uint32_t w_lo = static_cast<uint32_t>(desc), hi = static_cast<uint32_t>(desc >> 32), t0 = same_in_warp(tmem_base);
        int s = 0, round = 0;
        auto issue = [&](int kb) {
            const int group = kb / kSplitFlush, buf = group & 1;
            const bool first = kb % kSplitFlush == 0;
            if (first && group >= 2) { mbar_wait(acc_free + buf, ((group >> 1) - 1) & 1, p.err); tc_after(); }
            mbar_wait(full + s, round & 1, p.err);
            tc_after();
            const uint32_t wl = w_lo + s * (stage_bytes >> 4), al = wl + (3 * kSplitABytes >> 4), d = t0 + buf * 256, more0 = first ? 0u : 1u;
            constexpr uint32_t W1 = kSplitABytes >> 4, W2 = 2 * W1, A1 = b_plane >> 4, A2 = 2 * A1;
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < kSplitBK / 16; ++k) {
                    const uint32_t more = k > 0 ? 1u : more0;
                    auto at = [&](uint32_t lo) { return desc_words(lo + k * 2, hi); };
                    if (stacked) {                     // columns [0, NT): w0 a0;  [NT, 2 NT): w0 a1 + w1 a0;  [2 NT, 3 NT): w0 a2 + w1 a1 + w2 a0
                        umma(d, at(wl), at(al), id3, more);
                        umma(d + NT, at(wl + W1), at(al), id2, 1u);
                        umma(d + 2 * NT, at(wl + W2), at(al), id1, 1u);
                    } else {
                        umma(d, at(wl), at(al), id1, more);
                        umma(d + NT, at(wl + W2), at(al), id1, more);
                        umma(d + NT, at(wl + W1), at(al + A1), id1, 1u);
                        umma(d + NT, at(wl), at(al + A2), id1, 1u);
                        umma(d + NT, at(wl + W1), at(al), id1, 1u);
                        umma(d + NT, at(wl), at(al + A1), id1, 1u);
                    }
                }
                tc_commit(empty + s);
                if (kb % kSplitFlush == kSplitFlush - 1 || kb == num_kb - 1) tc_commit(acc_ready + buf);
            }
            __syncwarp();
            if (++s == STAGES) { s = 0; ++round; }
        };
        if (warp == 8) issue(0);
        uint64_t acc[COLS / 2];
#pragma unroll
        for (int j = 0; j < COLS / 2; ++j) acc[j] = 0;
        const uint32_t mine = tmem_base + half * COLS + (static_cast<uint32_t>(quarter * 32) << 16);
        for (int kb = 0; kb < num_kb; ++kb) {
            if (warp == 8 && kb + 1 < num_kb) issue(kb + 1);
            if (kb % kSplitFlush != kSplitFlush - 1 && kb != num_kb - 1) continue;
            __syncwarp();
            const int group = kb / kSplitFlush, buf = group & 1;
            mbar_wait(acc_ready + buf, (group >> 1) & 1, p.err);
            tc_after();
            const uint32_t d = mine + buf * 256;
#pragma unroll
            for (int j0 = 0; j0 < COLS; j0 += 16) {
                uint32_t u[16], v[16], t[16];
                if (stacked) tm_load16(d + 2 * NT + j0, t);
                tm_load16(d + NT + j0, v);
                tm_load16(d + j0, u);
                tm_wait_ld();
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                    uint64_t low = pack2(__uint_as_float(v[j]), __uint_as_float(v[j + 1]));
                    if (stacked) low = add2(low, pack2(__uint_as_float(t[j]), __uint_as_float(t[j + 1])));
                    acc[(j0 + j) / 2] = add2(acc[(j0 + j) / 2], add2(low, pack2(__uint_as_float(u[j]), __uint_as_float(u[j + 1]))));
                }
            }
            tc_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_free + buf);
        }
        if (gridDim.z == 1) {
            const int n = w0 + quarter * 32 + lane, first = m0 + half * COLS;
            if (n < p.N) {
#pragma unroll
                for (int j = 0; j < COLS; ++j)
                    if (first + j < p.M) split_store(p, first + j, n, __uint_as_float(static_cast<uint32_t>(j % 2 ? acc[j / 2] >> 32 : acc[j / 2])));
            }
        } else {                                       // all products have read the stages: the block's sums lie there for the cluster
            float* tile = reinterpret_cast<float*>(stage0) + (half * COLS) * kSplitRows + quarter * 32 + lane;
#pragma unroll
            for (int j = 0; j < COLS; ++j) tile[j * kSplitRows] = __uint_as_float(static_cast<uint32_t>(j % 2 ? acc[j / 2] >> 32 : acc[j / 2]));
        }
    }
    if (gridDim.z > 1) {                               // each block adds up and stores its rows of the tile, the parts of K in order
        __syncwarp();
        cluster_sync();
        const int n = threadIdx.x % kSplitRows;
        for (int j = blockIdx.z * 4 + threadIdx.x / kSplitRows; j < NT; j += gridDim.z * 4) {
            if (m0 + j >= p.M || w0 + n >= p.N) continue;
            const float* at = reinterpret_cast<const float*>(stage0) + j * kSplitRows + n;
            float v = ld_cluster(at, 0);
            for (int z = 1; z < static_cast<int>(gridDim.z); ++z) v += ld_cluster(at, z);
            split_store(p, m0 + j, w0 + n, v);
        }
        __syncwarp();
        cluster_sync();                                // no block leaves while another reads its sums
    }
    tc_before();
    __syncthreads();
    if (warp == 8) {
        tc_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512));
    }
}

template <int NT>
static int launch_split(const SplitParams& p, int parts, bool dependent, cudaStream_t stream) {
    constexpr int stages = NT <= kSplitStack ? 3 : 2;
    constexpr size_t smem = 1024 + static_cast<size_t>(stages) * 3 * (kSplitABytes + NT * 128) + 10 * 8 + 16;
    static bool set = false;
    if (!set) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_split_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return static_cast<int>(e);
        set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.N + kSplitRows - 1) / kSplitRows, (p.M + NT - 1) / NT, parts);
    cfg.blockDim = dim3(kSplitThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (parts > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 1;
        attr[n].val.clusterDim.y = 1;
        attr[n].val.clusterDim.z = parts;
        ++n;
    }
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (dependent && pdl_enabled() && cudaStreamIsCapturing(stream, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    cudaLaunchKernelEx(&cfg, gemm_f32_split_kernel<NT>, p);
    return launch_status();
}

}  // namespace cvb

using namespace cvb;

// tile: rows of A a block (32, 64, 96 or 128); parts: blocks that share a tile's K (1, 2, 4 or 8, each with 64 of K or more).
// dependent: launch with the programmatic-dependent-launch attribute (outside captures).
extern "C" int cvb_gemm_f32_split(float* out, const float* a, const float* w, int M, int N, int K, int tile, int parts, int dependent, int* err_flag,
                                  cudaStream_t stream) {
    if (M == 0) return CVB_OK;
    if (M < 0 || N <= 0 || K <= 0) return CVB_E_SIZE;
    if (tile < 32 || tile > 128 || tile % 32 || parts < 1 || parts > 8 || (parts & (parts - 1)) || parts > (K + kSplitBK - 1) / kSplitBK) return CVB_E_SHAPE;
    if (K % 4 || ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) != 0) return CVB_E_ALIGN;
    const int64_t rows = (static_cast<int64_t>(M) + tile - 1) / tile;
    if (rows > 65535) return CVB_E_SIZE;
    if ((static_cast<int64_t>(M) > N ? M : N) * static_cast<int64_t>(K) > (1LL << 30) - 1) return CVB_E_SIZE;     // byte offsets in 32 bits
    const SplitParams p{out, a, w, M, N, K, err_flag};
    if (tile == 32) return launch_split<32>(p, parts, dependent != 0, stream);
    if (tile == 64) return launch_split<64>(p, parts, dependent != 0, stream);
    if (tile == 96) return launch_split<96>(p, parts, dependent != 0, stream);
    return launch_split<128>(p, parts, dependent != 0, stream);
}
