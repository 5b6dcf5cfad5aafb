// The delta rule with one decay per head and token over prompt portions, in chunks of 32 tokens on the tensor cores:
//
//   S <- g_t S;  u_t = b_t (v_t - S^T k_t);  S <- S + k_t u_t^T;  o_t = S^T q_t          (recurrent.cu: delta_scan, one token after the other)
//
// The token-by-token scan is a chain: two reductions over a column of S per token, about 800 cycles a token whatever the number of heads
// (1,511 tokens, 16 heads of 128 x 128: 626 us).  With D_ij = g_{j+1} .. g_i (j <= i), e_i = g_0 .. g_i inside a chunk and S_0 the state
// in front of it, a chunk's tokens are one triangular system
//   (I + L) U = b (V - e K S_0),  L_ij = b_i D_ij (k_i . k_j) for j < i          W = (I + L)^-1 b e K,  U~ = (I + L)^-1 b V
//   U = U~ - W S_0;   O = e Q S_0 + A U,  A_ij = D_ij (q_i . k_j) for j <= i;     S = e_31 S_0 + K^T (D_31,j U_j)
// delta_prepare_kernel makes W, U~, A, e and D_31 of every (chunk, head) side by side; delta_chain_kernel walks the chunks of a
// (request, head, slice of value columns) with S in registers, two barriers and about 24 + 12 products a warp and chunk.  Decays are
// running products (never logarithms: g may be 0).
//
// Products run as `mma.sync.m16n8k16` with every float operand split into two bf16 (x = hi + lo, hi hi + hi lo + lo hi, float
// accumulation): 2^-17 of an operand is lost, 1 / 64 of what the bf16 projection in front of the rule has rounded already.  W and U~ come
// from a float substitution, one thread per column.  Steps in float32 stay on the scan.
// Chunk images in scratch are laid out as the chain kernel wants them in shared memory (rows padded against ldmatrix conflicts), so a
// chunk arrives by three bulk copies, two chunks ahead.  What bounds the chain: the mma.sync rate and the copies from the L2 (57 KB a
// chunk and block).
#include "common.cuh"
#include "sm100.cuh"
#include "mma_tiles.cuh"

namespace cvb {

constexpr int kDC = 32;                                  // tokens per chunk
constexpr int kDK = 128;                                 // key channels
constexpr int kDLD = kDK + 8;                            // bf16 elements of a padded row of K, Q, W
constexpr int kDLA = kDC + 8;                            // of A
constexpr int kDRowsBytes = kDC * kDLD * 2;              // one image of K, Q or W
constexpr int kDHeadBytes = 2 * kDRowsBytes + 2 * kDC * kDLA * 2 + 2 * kDC * 4;     // W hi, lo | A hi, lo | e | D_31
constexpr int kDKvBytes = 4 * kDRowsBytes;               // K hi, lo | Q hi, lo

struct DeltaChunkParams {
    const float* qn;                                     // [T, G * 128]
    const float* kn;
    const float* vv;                                     // [T, H * dv]
    const float* gg;                                     // [T, H]
    const float* bb;                                     // [T, H]
    float* out;                                          // [T, H * dv]
    float* state;
    int64_t state_floats;
    const int* cu_seqlens;
    const int* state_slots;
    int num_slots, S, H, G, dv;
    int c_first, c_count;                                // the chunks (of all requests in order) that the scratch holds now
    unsigned char* scratch;                              // [c_count][H][head image] | [c_count][G][kv image] | [c_count][H][dv / NB][32][NB + 8] float
    int* err;
};

__device__ __forceinline__ int chunks_of(const DeltaChunkParams& p, int s) { return (p.cu_seqlens[s + 1] - p.cu_seqlens[s] + kDC - 1) / kDC; }

__device__ __forceinline__ unsigned char* head_image(const DeltaChunkParams& p, int lc, int h) {
    return p.scratch + (static_cast<int64_t>(lc) * p.H + h) * kDHeadBytes;
}
__device__ __forceinline__ unsigned char* kv_image(const DeltaChunkParams& p, int lc, int g) {
    return p.scratch + static_cast<int64_t>(p.c_count) * p.H * kDHeadBytes + (static_cast<int64_t>(lc) * p.G + g) * kDKvBytes;
}
template <int NB>
__device__ __forceinline__ float* u_image(const DeltaChunkParams& p, int lc, int h, int cb) {
    unsigned char* base = p.scratch + static_cast<int64_t>(p.c_count) * (static_cast<int64_t>(p.H) * kDHeadBytes + static_cast<int64_t>(p.G) * kDKvBytes);
    return reinterpret_cast<float*>(base) + ((static_cast<int64_t>(lc) * p.H + h) * (p.dv / NB) + cb) * (kDC * (NB + 8));
}

__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16& hi, __nv_bfloat16& lo) {
    hi = __float2bfloat16_rn(x);
    lo = __float2bfloat16_rn(x - __bfloat162float(hi));
}
__device__ __forceinline__ void split_pair(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const float2 f = __bfloat1622float2(h);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = pack2(x - f.x, y - f.y);
}

// Grid (chunk, head), 128 + dv threads: thread c < 128 solves for column c of W, the others for a column of U~.
template <int NB>
__global__ void __launch_bounds__(256)
delta_prepare_kernel(const DeltaChunkParams p) {
    pdl_trigger();
    extern __shared__ __align__(128) unsigned char smem[];
    __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(smem);                    // hi, lo
    __nv_bfloat16* sQ = sK + 2 * kDC * kDLD;                                       // hi, lo
    float* sL = reinterpret_cast<float*>(sQ + 2 * kDC * kDLD);                     // L transposed: [j][i], rows of 36
    float* sD = sL + kDC * 36;                                                     // [i][j], rows of 33
    float* sG = sD + kDC * 33;                                                     // g, b, e
    float* sBeta = sG + kDC;
    float* sE = sBeta + kDC;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lc = blockIdx.x, h = blockIdx.y, share = p.H / p.G, kvh = h / share;
    // which request the chunk belongs to: the lanes of a warp take a request each (every warp does the same)
    const int chunk = p.c_first + lc;
    int seq = -1, ci = 0, before = 0;
    for (int s0 = 0; s0 < p.S && seq < 0; s0 += 32) {
        const int s = s0 + lane;
        const int n = s < p.S ? chunks_of(p, s) : 0;
        int upto = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const int first = before + upto - n;
        const unsigned hit = __ballot_sync(0xffffffffu, n > 0 && chunk >= first && chunk < first + n);
        if (hit) {
            const int src = __ffs(hit) - 1;
            seq = s0 + src;
            ci = chunk - __shfl_sync(0xffffffffu, first, src);
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (seq < 0) return;
    const int t0 = p.cu_seqlens[seq] + ci * kDC, n = min(kDC, p.cu_seqlens[seq + 1] - t0);
    pdl_wait();
    // tokens past the portion: k, q, v, b zero and g one, which leaves the state as it is
    for (int idx = tid; idx < 2 * kDC * (kDK / 4); idx += blockDim.x) {
        const int which = idx / (kDC * (kDK / 4)), r = idx / (kDK / 4) % kDC, c = idx % (kDK / 4) * 4;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < n) x = *reinterpret_cast<const float4*>((which ? p.qn : p.kn) + (static_cast<int64_t>(t0 + r) * p.G + kvh) * kDK + c);
        uint2 hi, lo;
        split_pair(x.x, x.y, hi.x, lo.x);
        split_pair(x.z, x.w, hi.y, lo.y);
        __nv_bfloat16* dst = (which ? sQ : sK) + r * kDLD + c;
        *reinterpret_cast<uint2*>(dst) = hi;
        *reinterpret_cast<uint2*>(dst + kDC * kDLD) = lo;
    }
    if (tid < kDC) {
        sG[tid] = tid < n ? p.gg[static_cast<int64_t>(t0 + tid) * p.H + h] : 1.f;
        sBeta[tid] = tid < n ? p.bb[static_cast<int64_t>(t0 + tid) * p.H + h] : 0.f;
    }
    // the thread's right-hand side, asked for now and used after the products
    const int col = tid < kDK ? tid : tid - kDK;
    const bool is_w = tid < kDK;
    float x[kDC];
#pragma unroll
    for (int i = 0; i < kDC; ++i) {
        const float* src = is_w ? p.kn + (static_cast<int64_t>(t0 + i) * p.G + kvh) * kDK + col : p.vv + (static_cast<int64_t>(t0 + i) * p.H + h) * p.dv + col;
        x[i] = i < n ? *src : 0.f;
    }
    __syncthreads();
    if (warp == 0) {                                                               // D, a column per lane
        float d = 1.f;
        for (int i = 0; i < kDC; ++i) {
            if (i > lane) d *= sG[i];
            sD[i * 33 + lane] = d;                                                 // read for j <= i only
        }
    } else if (warp == 1) {
        float e = 1.f;
        for (int s = 0; s <= lane; ++s) e *= sG[s];
        sE[lane] = e;
    }
    if (h % share == 0) {                                                          // the kv head's image, once
        const uint4* src = reinterpret_cast<const uint4*>(smem);
        uint4* dst = reinterpret_cast<uint4*>(kv_image(p, lc, kvh));
        for (int i = tid; i < kDKvBytes / 16; i += blockDim.x) dst[i] = src[i];
    }
    __syncthreads();
    unsigned char* img = head_image(p, lc, h);
    // K K^T and Q K^T: 2 x 2 x 4 tiles of 16 x 8 for eight warps (six, where a head's values are 64 wide: some warps take two)
    for (int tile = warp; tile < 8; tile += blockDim.x >> 5) {
        const int m = (tile & 1) * 16, nn = (tile >> 1) * 8;
        float kk[4] = {0.f, 0.f, 0.f, 0.f}, qk[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < kDK / 16; ++k) {
            const int ao = (m + (lane & 15)) * kDLD + k * 16 + (lane >> 4) * 8;
            uint32_t kh[4], kl[4], qh[4], ql[4], b[4];
            ldm_x4(kh, sK + ao); ldm_x4(kl, sK + kDC * kDLD + ao);
            ldm_x4(qh, sQ + ao); ldm_x4(ql, sQ + kDC * kDLD + ao);
            // b[0], b[1]: hi, columns k*16 and k*16 + 8 of the eight rows; b[2], b[3]: lo
            ldm_x4(b, sK + (lane >> 4) * kDC * kDLD + (nn + (lane & 7)) * kDLD + k * 16 + ((lane >> 3) & 1) * 8);
            mma_16816(kk, kh, b[0], b[1]); mma_16816(kk, kh, b[2], b[3]); mma_16816(kk, kl, b[0], b[1]);
            mma_16816(qk, qh, b[0], b[1]); mma_16816(qk, qh, b[2], b[3]); mma_16816(qk, ql, b[0], b[1]);
        }
        __nv_bfloat16* a_img = reinterpret_cast<__nv_bfloat16*>(img + 2 * kDRowsBytes);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int i = m + (lane >> 2) + half * 8, j = nn + (lane & 3) * 2;
            sL[j * 36 + i] = j < i ? sBeta[i] * sD[i * 33 + j] * kk[half * 2] : 0.f;
            sL[(j + 1) * 36 + i] = j + 1 < i ? sBeta[i] * sD[i * 33 + j + 1] * kk[half * 2 + 1] : 0.f;
            uint32_t hi, lo;
            split_pair(j <= i ? sD[i * 33 + j] * qk[half * 2] : 0.f, j + 1 <= i ? sD[i * 33 + j + 1] * qk[half * 2 + 1] : 0.f, hi, lo);
            *reinterpret_cast<uint32_t*>(a_img + i * kDLA + j) = hi;
            *reinterpret_cast<uint32_t*>(a_img + kDC * kDLA + i * kDLA + j) = lo;
        }
    }
    if (tid < kDC) {
        float* v = reinterpret_cast<float*>(img + 2 * kDRowsBytes + 2 * kDC * kDLA * 2);
        v[tid] = sE[tid];
        v[kDC + tid] = sD[(kDC - 1) * 33 + tid];
    }
    __syncthreads();
    // forward substitution, column by column of L: x_i -= L_ij x_j
#pragma unroll
    for (int i = 0; i < kDC; ++i) x[i] *= is_w ? sBeta[i] * sE[i] : sBeta[i];
#pragma unroll
    for (int j = 0; j < kDC - 1; ++j) {
#pragma unroll
        for (int i4 = (j + 1) / 4 * 4; i4 < kDC; i4 += 4) {
            const float4 l = *reinterpret_cast<const float4*>(sL + j * 36 + i4);   // zero on and above the diagonal
            x[i4] = fmaf(-l.x, x[j], x[i4]);
            x[i4 + 1] = fmaf(-l.y, x[j], x[i4 + 1]);
            x[i4 + 2] = fmaf(-l.z, x[j], x[i4 + 2]);
            x[i4 + 3] = fmaf(-l.w, x[j], x[i4 + 3]);
        }
    }
    if (is_w) {
        __nv_bfloat16* w = reinterpret_cast<__nv_bfloat16*>(img);
#pragma unroll
        for (int i = 0; i < kDC; ++i) {
            __nv_bfloat16 hi, lo;
            split_bf16(x[i], hi, lo);
            w[i * kDLD + col] = hi;
            w[kDC * kDLD + i * kDLD + col] = lo;
        }
    } else {
        float* u = u_image<NB>(p, lc, h, col / NB) + col % NB;
#pragma unroll
        for (int i = 0; i < kDC; ++i) u[i * (NB + 8)] = x[i];
    }
}

template <int NB>
struct DeltaChainSmem {
    static constexpr int kU = kDC * (NB + 8) * 4;
    static constexpr int kStage = kDHeadBytes + kDKvBytes + kU;
    static constexpr int kS = 2 * kDK * (NB + 8) * 2;                              // S hi, lo
    static constexpr int kUb = 4 * kDC * (NB + 8) * 2;                             // U hi, lo | D U hi, lo
    static constexpr size_t kBytes = static_cast<size_t>(2) * kStage + kS + kUb + 2 * 8;
};

// Grid (request, head, NB value columns); NB / 2 warps: one half makes W S, the other Q S (tiles of 16 x 8), then every warp two tiles of S.
template <int NB>
__global__ void __launch_bounds__(NB * 16, 1)
delta_chain_kernel(const DeltaChunkParams p) {
    pdl_trigger();
    extern __shared__ __align__(128) unsigned char smem[];
    using L = DeltaChainSmem<NB>;
    constexpr int LS = NB + 8, kWarps = NB / 2, kHalf = kWarps / 2;
    unsigned char* sStage = smem;
    __nv_bfloat16* sS = reinterpret_cast<__nv_bfloat16*>(smem + 2 * L::kStage);
    __nv_bfloat16* sU = sS + 2 * kDK * LS;
    __nv_bfloat16* sDU = sU + 2 * kDC * LS;
    uint64_t* full = reinterpret_cast<uint64_t*>(sDU + 2 * kDC * LS);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int s = blockIdx.x, h = blockIdx.y, cb = blockIdx.z, kvh = h / (p.H / p.G);
    const int slot = p.state_slots[s];
    if (slot < 0 || slot >= p.num_slots) {
        if (tid == 0) atomicExch(p.err, 2);
        return;
    }
    int first = 0;                                                                 // the request's first chunk among all
    for (int r = lane; r < s; r += 32) first += chunks_of(p, r);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) first += __shfl_xor_sync(0xffffffffu, first, o);
    const int begin = p.cu_seqlens[s], end = p.cu_seqlens[s + 1];
    const int c0 = max(first, p.c_first), c1 = min(first + chunks_of(p, s), p.c_first + p.c_count);
    if (c0 >= c1) return;
    if (tid == 0) {
        mbar_init(full, 1);
        mbar_init(full + 1, 1);
        mbar_fence_init();
    }
    pdl_wait();
    auto fetch = [&](int c) {                                                      // one thread: chunk c into its stage
        const int st = (c - c0) & 1, lc = c - p.c_first;
        unsigned char* dst = sStage + st * L::kStage;
        mbar_expect_tx(full + st, L::kStage);
        const void* src[3] = {head_image(p, lc, h), kv_image(p, lc, kvh), u_image<NB>(p, lc, h, cb)};
        const int bytes[3] = {kDHeadBytes, kDKvBytes, L::kU};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                         ::"r"(smem_u32(dst)), "l"(src[i]), "r"(bytes[i]), "r"(smem_u32(full + st)) : "memory");
            dst += bytes[i];
        }
    };
    if (tid == 0) {
        fetch(c0);
        if (c0 + 1 < c1) fetch(c0 + 1);
    }
    // S: this warp's two tiles of 16 rows x 8 columns
    const int sm = (NB == 16 ? warp : warp & 7) * 16, sn = NB == 16 ? 0 : (warp >> 3) * 16;
    float* st_base = p.state + static_cast<int64_t>(slot) * p.state_floats + static_cast<int64_t>(h) * kDK * p.dv + cb * NB;
    float S[2][4];
    auto write_s = [&]() {
#pragma unroll
        for (int t = 0; t < 2; ++t) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t hi, lo;
                split_pair(S[t][half * 2], S[t][half * 2 + 1], hi, lo);
                __nv_bfloat16* dst = sS + (sm + (lane >> 2) + half * 8) * LS + sn + t * 8 + (lane & 3) * 2;
                *reinterpret_cast<uint32_t*>(dst) = hi;
                *reinterpret_cast<uint32_t*>(dst + kDK * LS) = lo;
            }
        }
    };
#pragma unroll
    for (int t = 0; t < 2; ++t) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const float2 v = *reinterpret_cast<const float2*>(st_base + static_cast<int64_t>(sm + (lane >> 2) + half * 8) * p.dv + sn + t * 8 + (lane & 3) * 2);
            S[t][half * 2] = v.x;
            S[t][half * 2 + 1] = v.y;
        }
    }
    write_s();
    __syncthreads();
    const bool is_q = warp >= kHalf;
    const int w = is_q ? warp - kHalf : warp, m = (w & 1) * 16, nn = (w >> 1) * 8;
    for (int c = c0; c < c1; ++c) {
        const int st = (c - c0) & 1;
        const unsigned char* base = sStage + st * L::kStage;
        const __nv_bfloat16* sW = reinterpret_cast<const __nv_bfloat16*>(base);
        const __nv_bfloat16* sA = sW + 2 * kDC * kDLD;
        const float* sE = reinterpret_cast<const float*>(sA + 2 * kDC * kDLA);
        const __nv_bfloat16* sK = reinterpret_cast<const __nv_bfloat16*>(base + kDHeadBytes);
        const __nv_bfloat16* sQ = sK + 2 * kDC * kDLD;
        const float* sUt = reinterpret_cast<const float*>(base + kDHeadBytes + kDKvBytes);
        mbar_wait(full + st, ((c - c0) >> 1) & 1, p.err);
        // W S (first half of the warps) or Q S: chains of their own for the three parts of the split
        float a0[4] = {0.f, 0.f, 0.f, 0.f}, a1[4] = {0.f, 0.f, 0.f, 0.f}, a2[4] = {0.f, 0.f, 0.f, 0.f};
        const __nv_bfloat16* lhs = (is_q ? sQ : sW) + (m + (lane & 15)) * kDLD + (lane >> 4) * 8;
        const __nv_bfloat16* rhs = sS + lane * LS + nn;
#pragma unroll
        for (int k = 0; k < kDK / 16; k += 2) {
            uint32_t bh[4], bl[4];
            ldm_x4_trans(bh, rhs + k * 16 * LS);
            ldm_x4_trans(bl, rhs + (kDK + k * 16) * LS);
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
                uint32_t xh[4], xl[4];
                ldm_x4(xh, lhs + (k + kk) * 16);
                ldm_x4(xl, lhs + kDC * kDLD + (k + kk) * 16);
                mma_16816(a0, xh, bh[2 * kk], bh[2 * kk + 1]);
                mma_16816(a1, xh, bl[2 * kk], bl[2 * kk + 1]);
                mma_16816(a2, xl, bh[2 * kk], bh[2 * kk + 1]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) a0[i] += a1[i] + a2[i];
        if (!is_q) {                                                               // U = U~ - W S, and D_31 U
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int i = m + (lane >> 2) + half * 8, j = nn + (lane & 3) * 2;
                const float2 ut = *reinterpret_cast<const float2*>(sUt + i * LS + j);
                const float ux = ut.x - a0[half * 2], uy = ut.y - a0[half * 2 + 1], d = sE[kDC + i];
                uint32_t hi, lo;
                split_pair(ux, uy, hi, lo);
                *reinterpret_cast<uint32_t*>(sU + i * LS + j) = hi;
                *reinterpret_cast<uint32_t*>(sU + (kDC + i) * LS + j) = lo;
                split_pair(d * ux, d * uy, hi, lo);
                *reinterpret_cast<uint32_t*>(sDU + i * LS + j) = hi;
                *reinterpret_cast<uint32_t*>(sDU + (kDC + i) * LS + j) = lo;
            }
        }
        __syncthreads();                                                           // U is there; nobody reads the old S any more
        {                                                                          // S = e_31 S + K^T (D_31 U)
            const float e = sE[kDC - 1];
            float acc[2][4];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[t][i] = 0.f;
            }
            const int ko = ((lane & 7) + (lane >> 4) * 8) * kDLD + sm + ((lane >> 3) & 1) * 8;
            uint32_t bh[2][4], bl[2][4];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                ldm_x4_trans(bh[t], sDU + lane * LS + sn + t * 8);
                ldm_x4_trans(bl[t], sDU + (kDC + lane) * LS + sn + t * 8);
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                uint32_t kh[4], kl[4];
                ldm_x4_trans(kh, sK + k * 16 * kDLD + ko);
                ldm_x4_trans(kl, sK + (kDC + k * 16) * kDLD + ko);
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    mma_16816(acc[t], kh, bh[t][2 * k], bh[t][2 * k + 1]);
                    mma_16816(acc[t], kh, bl[t][2 * k], bl[t][2 * k + 1]);
                    mma_16816(acc[t], kl, bh[t][2 * k], bh[t][2 * k + 1]);
                }
            }
#pragma unroll
            for (int t = 0; t < 2; ++t) {
#pragma unroll
                for (int i = 0; i < 4; ++i) S[t][i] = fmaf(e, S[t][i], acc[t][i]);
            }
            if (c + 1 < c1) write_s();
        }
        if (is_q) {                                                                // O = e Q S + A U
            float o[4];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const float e = sE[m + (lane >> 2) + half * 8];
                o[half * 2] = e * a0[half * 2];
                o[half * 2 + 1] = e * a0[half * 2 + 1];
            }
            uint32_t bh[4], bl[4];
            ldm_x4_trans(bh, sU + lane * LS + nn);
            ldm_x4_trans(bl, sU + (kDC + lane) * LS + nn);
            const __nv_bfloat16* al = sA + (m + (lane & 15)) * kDLA + (lane >> 4) * 8;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                uint32_t xh[4], xl[4];
                ldm_x4(xh, al + k * 16);
                ldm_x4(xl, al + kDC * kDLA + k * 16);
                mma_16816(o, xh, bh[2 * k], bh[2 * k + 1]);
                mma_16816(o, xh, bl[2 * k], bl[2 * k + 1]);
                mma_16816(o, xl, bh[2 * k], bh[2 * k + 1]);
            }
            const int t0 = begin + (c - first) * kDC;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int t = t0 + m + (lane >> 2) + half * 8;
                if (t < end)
                    *reinterpret_cast<float2*>(p.out + (static_cast<int64_t>(t) * p.H + h) * p.dv + cb * NB + nn + (lane & 3) * 2) = make_float2(o[half * 2], o[half * 2 + 1]);
            }
        }
        __syncthreads();                                                           // the new S is there; the stage may be filled again
        if (tid == 0 && c + 2 < c1) fetch(c + 2);
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
#pragma unroll
        for (int half = 0; half < 2; ++half)
            *reinterpret_cast<float2*>(st_base + static_cast<int64_t>(sm + (lane >> 2) + half * 8) * p.dv + sn + t * 8 + (lane & 3) * 2) =
                make_float2(S[t][half * 2], S[t][half * 2 + 1]);
    }
}

template <int NB>
int64_t delta_chunk_bytes(int H, int G, int dv) {
    return static_cast<int64_t>(H) * kDHeadBytes + static_cast<int64_t>(G) * kDKvBytes + static_cast<int64_t>(H) * (dv / NB) * kDC * (NB + 8) * 4;
}

template <int NB>
int launch_delta_chunks(DeltaChunkParams p, int total, int held, cudaStream_t stream) {
    const size_t prep = static_cast<size_t>(kDKvBytes) + (kDC * 36 + kDC * 33 + 3 * kDC) * sizeof(float);
    static bool set = false;
    if (!set) {
        if (cudaFuncSetAttribute(delta_prepare_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(prep)) != cudaSuccess ||
            cudaFuncSetAttribute(delta_chain_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(DeltaChainSmem<NB>::kBytes)) != cudaSuccess)
            return launch_status();
        set = true;
    }
    // a step of more chunks than the scratch holds goes through it in several turns; the state carries on from one to the next
    for (int c = 0; c < total; c += held) {
        p.c_first = c;
        p.c_count = total - c < held ? total - c : held;
        launch_kernel(delta_prepare_kernel<NB>, dim3(p.c_count, p.H), dim3(kDK + p.dv), prep, stream, p);
        launch_kernel(delta_chain_kernel<NB>, dim3(p.S, p.H, p.dv / NB), dim3(NB * 16), DeltaChainSmem<NB>::kBytes, stream, p);
    }
    return launch_status();
}

}  // namespace cvb

using namespace cvb;

// Bytes of scratch for `chunks` chunks (of 32 tokens); slices of 16 value columns need the most.
extern "C" int64_t cvb_delta_chunks_scratch(int chunks, int H, int G, int dv) { return static_cast<int64_t>(chunks) * delta_chunk_bytes<16>(H, G, dv); }

// total: the sum over the requests of ceil(tokens / 32).
extern "C" int cvb_delta_chunks(float* out, const float* qn, const float* kn, const float* vv, const float* gg, const float* bb, float* state,
                                int64_t state_floats, const int* cu_seqlens, const int* state_slots, int num_slots, int S, int total, int H, int G,
                                int dk, int dv, void* scratch, int64_t scratch_bytes, int* err_flag, cudaStream_t stream) {
    if (S == 0 || total == 0) return CVB_OK;
    if (S < 0 || total < 0 || H <= 0 || H > 65535 || G <= 0 || num_slots <= 0) return CVB_E_SIZE;
    if (dk != kDK || (dv != 64 && dv != 128)) return CVB_E_UNSUPPORTED;
    if (H % G || state_floats < static_cast<int64_t>(H) * dk * dv) return CVB_E_SHAPE;
    for (const void* p : {static_cast<const void*>(qn), static_cast<const void*>(kn), static_cast<const void*>(vv), static_cast<const void*>(out),
                          static_cast<const void*>(state), static_cast<const void*>(scratch)})
        if (reinterpret_cast<uintptr_t>(p) & 15) return CVB_E_ALIGN;
    if (state_floats % 2) return CVB_E_ALIGN;                                      // a slot's matrices start on whole pairs
    DeltaChunkParams p{};
    p.qn = qn; p.kn = kn; p.vv = vv; p.gg = gg; p.bb = bb; p.out = out; p.state = state; p.state_floats = state_floats;
    p.cu_seqlens = cu_seqlens; p.state_slots = state_slots; p.num_slots = num_slots; p.S = S; p.H = H; p.G = G; p.dv = dv;
    p.scratch = static_cast<unsigned char*>(scratch); p.err = err_flag;
    // slices of 16 columns while the chain's blocks fit the SMs at once (each holds an SM's shared memory), else of 32
    const bool narrow = static_cast<int64_t>(S) * H * (dv / 16) <= 148;
    const int64_t per = narrow ? delta_chunk_bytes<16>(H, G, dv) : delta_chunk_bytes<32>(H, G, dv);
    const int64_t held = scratch_bytes / per;
    if (held < 1) return CVB_E_SCRATCH;
    const int h32 = static_cast<int>(held < total ? held : total);
    return narrow ? launch_delta_chunks<16>(p, total, h32, stream) : launch_delta_chunks<32>(p, total, h32, stream);
}
