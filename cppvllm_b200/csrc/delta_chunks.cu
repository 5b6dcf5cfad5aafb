// The delta rule with one decay per head and token over prompt portions, in chunks of 32 tokens on the tensor cores:
//
//   S <- g_t S;  u_t = b_t (v_t - S^T k_t);  S <- S + k_t u_t^T;  o_t = S^T q_t          (recurrent.cu: delta_scan, one token after the other)
//
// The token-by-token scan is a chain: two reductions over a column of S per token, about 800 cycles a token whatever the number of heads
// (1,511 tokens, 16 heads of 128 x 128: 626 us).  With D_ij = g_{j+1} .. g_i (j <= i), e_i = g_0 .. g_i inside a chunk and S_0 the state
// in front of it, a chunk's tokens are one triangular system
//   (I + L) U = b (V - e K S_0),  L_ij = b_i D_ij (k_i . k_j) for j < i          W = (I + L)^-1 b e K,  U~ = (I + L)^-1 b V
//   U = U~ - W S_0;   O = e Q S_0 + A U,  A_ij = D_ij (q_i . k_j) for j <= i;     S = e_31 S_0 + K^T (D_31,j U_j)
// delta_prepare_kernel makes W, U~, A, e and D_31 of every (chunk, head) side by side, from the packed projection; delta_chain_kernel walks the chunks of a
// (request, head, slice of value columns) with S in registers, half of its warps on the chain and half on the outputs beside it.  Decays are
// running products (never logarithms: g may be 0).
//
// Products run as `mma.sync.m16n8k8` in tf32 with every float operand split in two when its fragment is loaded (x = hi + lo: hi the nearest tf32
// number, lo the rest, of which the product reads 11 bits more; hi hi + hi lo + lo hi), float accumulation, the leading terms in chains of two
// products that are added up by the float units (the tensor core cuts a sum off instead of rounding it; chains of four cost the outputs 4 %).  From
// the same projection, 64 to 2,048 tokens at 16/8 and 32/8 heads, the outputs are 2.5e-7 to 3.8e-7 from float64 and the states 2.4e-7 to 4.0e-7 (the
// float scan: 1.9e-7 to 3.7e-7, 2.2e-7 to 4.0e-7; with bf16 pairs 5.3e-6 to 6.3e-6, 4.7e-6 to 4.9e-6); behind the layer's bf16 projections the two
// routes are equally far, 4.2e-3.  W and U~ come from a float substitution, one thread per column.  Steps in float32 stay on the scan.
// Chunk images in scratch are laid out as the chain kernel wants them in shared memory (every operand with its inner dimension running, rows
// padded against ldmatrix conflicts), so a chunk arrives by a few bulk copies, two chunks ahead.
#include "common.cuh"
#include "sm100.cuh"
#include "mma_tiles.cuh"

namespace cvb {

constexpr int kDC = 32;                                  // tokens per chunk
constexpr int kDK = 128;                                 // key channels
constexpr int kDLF = kDK + 4;                            // floats of a padded row of K, Q, W, of convolved channels and of S transposed
constexpr int kDLT = kDC + 4;                            // floats of a padded row of A and of K, U, D U transposed
constexpr int kDRowsBytes = kDC * kDLF * 4;              // Q or W
constexpr int kDTransBytes = kDK * kDLT * 4;             // K transposed
constexpr int kDABytes = kDC * kDLT * 4;
constexpr int kDVecBytes = 2 * kDC * 4;
constexpr int kDHeadBytes = kDRowsBytes + kDABytes + kDVecBytes;                   // W | A | e | D_31
constexpr int kDKvBytes = kDTransBytes + kDRowsBytes;    // K transposed | Q

struct DeltaChunkParams {
    const __nv_bfloat16* packed;                         // rows of `stride` elements; from column qkv_off on q [G * 128], k [G * 128], v [H * dv]
    int stride, qkv_off;
    const float* conv_w;                                 // [channels, taps]
    const float* ba;                                     // [T, 2 H]: the input strengths' logits, then the decays'
    const float* dt_bias;                                // [H]
    const float* a_log;
    int64_t conv_off;                                    // where the convolution's history lies in a slot
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

// x = hi + lo: hi x rounded to tf32 (10 bits behind the first one), lo what is left, exact in float, of which the product reads its upper 11 bits.
// (Rounding lo instead of leaving its tail to be cut off changed no error by 1 % and cost 3 % of the rule.)  A NaN stays one in lo.
__device__ __forceinline__ void split_tf32(uint32_t x, uint32_t& hi, uint32_t& lo) {
    hi = (x + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(__uint_as_float(x) - __uint_as_float(hi));
}
template <int N>
__device__ __forceinline__ void split_tf32(const uint32_t (&x)[N], uint32_t (&hi)[N], uint32_t (&lo)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) split_tf32(x[i], hi[i], lo[i]);
}
// D += A B, 16 x 8 x 8.  With ldm_x4 over rows of floats a thread holds A's rows lane / 4 and + 8 at columns lane % 4 and + 4, and of B, whose
// columns are rows in memory, column lane / 4 at inner indices lane % 4, + 4 (and + 8, + 12: the next product's).
__device__ __forceinline__ void mma_1688(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// where a lane's rows lie for ldm_x4: of A 16 rows of 8 floats, of B 8 rows of 16
__device__ __forceinline__ int a_lane(int lane, int ld) { return (lane & 15) * ld + (lane >> 4) * 4; }
__device__ __forceinline__ int b_lane(int lane, int ld) { return (lane & 7) * ld + (lane >> 3) * 4; }

__device__ __forceinline__ float delta_sigmoid(float z) { return 1.f / (1.f + expf(-z)); }

constexpr int kDPair = 2;                                // heads of a kv head worked on together
constexpr size_t kDPrepBytes = static_cast<size_t>(4) * kDC * kDLF * sizeof(float) + kDPair * (kDC * 36 + kDC * 33 + 2 * kDC) * sizeof(float);

// Grid (chunk, kv head).  From the packed projection: convolutions, silu, unit vectors, decays and input strengths as recurrent.cu's delta_prep
// makes them, then the kv head's image and, two heads at a time, the heads' images; nothing between the projection and the images travels
// through memory.  (With delta_prep in front, a block per (chunk, head) and the heads' float rows read back, it was 66 + 49 us for 2,048
// tokens of 16/8 heads; now 59, bound by instruction issue with two blocks an SM.)
template <int NB, int TAPS>
__global__ void __launch_bounds__(256)
delta_prepare_kernel(const DeltaChunkParams p) {
    pdl_trigger();
    extern __shared__ __align__(128) unsigned char smem[];
    float* sK = reinterpret_cast<float*>(smem);                                    // k, convolved, then of unit length
    float* sQ = sK + kDC * kDLF;                                                   // q, the same
    float* sV0 = sQ + kDC * kDLF;
    float* sV1 = sV0 + kDC * kDLF;                                                 // the second head's v
    float* sL = sV1 + kDC * kDLF;                                                  // [head of the pair] L transposed: [j][i], rows of 36
    float* sD = sL + kDPair * kDC * 36;                                            // [i][j], rows of 33
    float* sG = sD + kDPair * kDC * 33;                                            // [head][b | e][32]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lc = blockIdx.x, kvh = blockIdx.y, share = p.H / p.G;
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
    const int slot = p.state_slots[seq];
    if (slot < 0 || slot >= p.num_slots) {
        if (tid == 0) atomicExch(p.err, 2);
        return;
    }
    const int QK = p.G * kDK, C = 2 * QK + p.H * p.dv;
    const float* hist = p.state + static_cast<int64_t>(slot) * p.state_floats + p.conv_off;
    pdl_wait();
    // Two neighbouring channels of eight tokens per thread.  The rows of all channels are asked for first, without a branch between them (a load in a
    // branch of its own is waited for there: eleven trips to memory, one after the other); rows past the portion stand in for themselves with its
    // first one and count as zeros.
    const int cp = (tid & 63) * 2, r0 = (tid >> 6) * 8;
    constexpr int kRows = 8 + TAPS - 1;
    auto fetch = [&](uint32_t (&raw)[kRows], float (&w)[2 * TAPS], int c0, int width) {      // w: [channel][tap]
        const int c = c0 + (cp < width ? cp : 0);
#pragma unroll
        for (int i = 0; i < 2 * TAPS; ++i) w[i] = p.conv_w[static_cast<int64_t>(c) * TAPS + i];
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            const int r = r0 + i - (TAPS - 1);                                     // the token's place in the chunk
            const bool in = r < n && ci * kDC + r >= 0;
            raw[i] = *reinterpret_cast<const uint32_t*>(p.packed + static_cast<int64_t>(t0 + (in ? r : 0)) * p.stride + p.qkv_off + c);
        }
    };
    auto convolve = [&](float* dst, const uint32_t (&raw)[kRows], const float (&w)[2 * TAPS], int c0, int width) {
        if (cp >= width) return;
        float2 x[kRows];
#pragma unroll
        for (int i = 0; i < kRows; ++i) x[i] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[i]));
        if (ci == 0 && r0 == 0) {                                                  // before the portion: the request's history, oldest first
#pragma unroll
            for (int i = 0; i < TAPS - 1; ++i) {
                x[i].x = hist[static_cast<int64_t>(i) * C + c0 + cp];
                x[i].y = hist[static_cast<int64_t>(i) * C + c0 + cp + 1];
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float ax = 0.f, ay = 0.f;
#pragma unroll
            for (int j = 0; j < TAPS; ++j) {
                ax = fmaf(w[j], x[i + j].x, ax);
                ay = fmaf(w[TAPS + j], x[i + j].y, ay);
            }
            const bool in = r0 + i < n;
            *reinterpret_cast<float2*>(dst + (r0 + i) * kDLF + cp) = make_float2(in ? ax / (1.f + expf(-ax)) : 0.f, in ? ay / (1.f + expf(-ay)) : 0.f);
        }
    };
    const int v_col = 2 * QK + kvh * share * p.dv;
    uint32_t raw_v1[kRows];
    float w_v1[2 * TAPS];
    {
        uint32_t raw_q[kRows], raw_k[kRows], raw_v[kRows];
        float w_q[2 * TAPS], w_k[2 * TAPS], w_v[2 * TAPS];
        fetch(raw_q, w_q, kvh * kDK, kDK);
        fetch(raw_k, w_k, QK + kvh * kDK, kDK);
        fetch(raw_v, w_v, v_col, p.dv);
        if (share > 1) fetch(raw_v1, w_v1, v_col + p.dv, p.dv);
        convolve(sQ, raw_q, w_q, kvh * kDK, kDK);
        convolve(sK, raw_k, w_k, QK + kvh * kDK, kDK);
        convolve(sV0, raw_v, w_v, v_col, p.dv);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kDC / 8; ++i) {                                            // unit vectors; a warp per row
        const int r = warp * (kDC / 8) + i;
#pragma unroll
        for (int which = 0; which < 2; ++which) {
            float* row = (which ? sQ : sK) + r * kDLF + lane * 4;
            const float4 x = *reinterpret_cast<const float4*>(row);
            const float ss = warp_sum(fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, x.w * x.w))));
            float inv = 1.f / sqrtf(ss + 1e-6f);
            if (which) inv *= 1.f / sqrtf(static_cast<float>(kDK));
            *reinterpret_cast<float4*>(row) = make_float4(x.x * inv, x.y * inv, x.z * inv, x.w * inv);
        }
    }
    __syncthreads();
    {                                                                              // the rows' pads are never read
        float* kt = reinterpret_cast<float*>(kv_image(p, lc, kvh));
        const int c = tid & (kDK - 1);
#pragma unroll
        for (int t = (tid >> 7) * 4; t < kDC; t += 8)
            *reinterpret_cast<float4*>(kt + c * kDLT + t) = make_float4(sK[t * kDLF + c], sK[(t + 1) * kDLF + c], sK[(t + 2) * kDLF + c], sK[(t + 3) * kDLF + c]);
        const uint4* src = reinterpret_cast<const uint4*>(sQ);
        uint4* dst = reinterpret_cast<uint4*>(kt + kDK * kDLT);
        for (int i = tid; i < kDRowsBytes / 16; i += 256) dst[i] = src[i];
    }
    // K K^T and Q K^T, one tile of 16 x 8 of either per warp, the same for all heads of the group
    const int m = (warp & 1) * 16, nn = (warp >> 1) * 8;
    float kk[4], qk[4];
    {
        float xk[4] = {0.f, 0.f, 0.f, 0.f}, xq[4] = {0.f, 0.f, 0.f, 0.f};          // the cross terms
#pragma unroll
        for (int i = 0; i < 4; ++i) kk[i] = qk[i] = 0.f;
#pragma unroll
        for (int k = 0; k < kDK / 16; ++k) {
            uint32_t b[4], bh[4], bl[4];
            ldm_x4(b, sK + nn * kDLF + k * 16 + b_lane(lane, kDLF));
            split_tf32(b, bh, bl);
            float ck[4] = {0.f, 0.f, 0.f, 0.f}, cq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                uint32_t a[4], ah[4], al[4];
                ldm_x4(a, sK + m * kDLF + k * 16 + e * 8 + a_lane(lane, kDLF));
                split_tf32(a, ah, al);
                mma_1688(ck, ah, bh[2 * e], bh[2 * e + 1]);
                mma_1688(xk, ah, bl[2 * e], bl[2 * e + 1]);
                mma_1688(xk, al, bh[2 * e], bh[2 * e + 1]);
                ldm_x4(a, sQ + m * kDLF + k * 16 + e * 8 + a_lane(lane, kDLF));
                split_tf32(a, ah, al);
                mma_1688(cq, ah, bh[2 * e], bh[2 * e + 1]);
                mma_1688(xq, ah, bl[2 * e], bl[2 * e + 1]);
                mma_1688(xq, al, bh[2 * e], bh[2 * e + 1]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) { kk[i] += ck[i]; qk[i] += cq[i]; }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) { kk[i] += xk[i]; qk[i] += xq[i]; }
    }
    for (int h0 = 0; h0 < share; h0 += kDPair) {
        const int heads = min(kDPair, share - h0), hbase = kvh * share + h0;
        const int c0 = v_col + h0 * p.dv;
        if (h0 > 0) {
            uint32_t raw[kRows];
            float w[2 * TAPS];
            fetch(raw, w, c0, p.dv);
            if (heads > 1) fetch(raw_v1, w_v1, c0 + p.dv, p.dv);
            convolve(sV0, raw, w, c0, p.dv);
        }
        if (heads > 1) convolve(sV1, raw_v1, w_v1, c0 + p.dv, p.dv);
        if (warp < heads) {                                                        // a head per warp, a token per lane
            const int h = hbase + warp;
            float g = 1.f, be = 0.f;
            if (lane < n) {
                const float* ba = p.ba + static_cast<int64_t>(t0 + lane) * 2 * p.H + h;
                const float z = ba[p.H] + p.dt_bias[h], sp = z > 20.f ? z : log1pf(expf(z));
                g = expf(-expf(p.a_log[h]) * sp);
                be = delta_sigmoid(ba[0]);
            }
            float* G = sG + warp * 2 * kDC;
            G[lane] = be;
            float d = 1.f, e = 1.f, mine = 1.f;                                    // D_i,lane and e_i: running products
#pragma unroll
            for (int i = 0; i < kDC; ++i) {
                const float gi = __shfl_sync(0xffffffffu, g, i);
                e *= gi;
                if (i > lane) d *= gi;
                if (i == lane) mine = e;
                sD[warp * kDC * 33 + i * 33 + lane] = d;                           // read for j <= i only
            }
            G[kDC + lane] = mine;
        }
        __syncthreads();
        for (int x = 0; x < heads; ++x) {
            unsigned char* img = head_image(p, lc, hbase + x);
            float* a_img = reinterpret_cast<float*>(img + kDRowsBytes);
            const float* D = sD + x * kDC * 33;
            const float* G = sG + x * 2 * kDC;
            float* Lt = sL + x * kDC * 36;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int i = m + (lane >> 2) + half * 8, j = nn + (lane & 3) * 2;
                Lt[j * 36 + i] = j < i ? G[i] * D[i * 33 + j] * kk[half * 2] : 0.f;
                Lt[(j + 1) * 36 + i] = j + 1 < i ? G[i] * D[i * 33 + j + 1] * kk[half * 2 + 1] : 0.f;
                *reinterpret_cast<float2*>(a_img + i * kDLT + j) = make_float2(j <= i ? D[i * 33 + j] * qk[half * 2] : 0.f,
                                                                               j + 1 <= i ? D[i * 33 + j + 1] * qk[half * 2 + 1] : 0.f);
            }
            if (tid < kDC) {
                float* v = reinterpret_cast<float*>(img + kDRowsBytes + kDABytes);
                v[tid] = G[kDC + tid];
                v[kDC + tid] = D[(kDC - 1) * 33 + tid];
            }
        }
        __syncthreads();
        // forward substitution, column by column of L: x_i -= L_ij x_j; threads 0 .. 127 a column of W, the others of U~
        const bool is_w = tid < kDK;
        const int col = tid & (kDK - 1);
        for (int x2 = 0; x2 < heads; ++x2) {
            if (!is_w && col >= p.dv) continue;
            const float* Lt = sL + x2 * kDC * 36;
            const float* G = sG + x2 * 2 * kDC;
            const float* rhs = (is_w ? sK : (x2 ? sV1 : sV0)) + col;
            float x[kDC];
#pragma unroll
            for (int i = 0; i < kDC; ++i) x[i] = rhs[i * kDLF] * (is_w ? G[i] * G[kDC + i] : G[i]);
#pragma unroll
            for (int j = 0; j < kDC - 1; ++j) {
#pragma unroll
                for (int i4 = (j + 1) / 4 * 4; i4 < kDC; i4 += 4) {
                    const float4 l = *reinterpret_cast<const float4*>(Lt + j * 36 + i4);
                    if (i4 > j) x[i4] = fmaf(-l.x, x[j], x[i4]);                       // rows up to j stay out of it: 0 times a bad x_j is a NaN
                    if (i4 + 1 > j) x[i4 + 1] = fmaf(-l.y, x[j], x[i4 + 1]);
                    if (i4 + 2 > j) x[i4 + 2] = fmaf(-l.z, x[j], x[i4 + 2]);
                    x[i4 + 3] = fmaf(-l.w, x[j], x[i4 + 3]);
                }
            }
            if (is_w) {
                float* w = reinterpret_cast<float*>(head_image(p, lc, hbase + x2)) + col;
#pragma unroll
                for (int i = 0; i < kDC; ++i) w[i * kDLF] = x[i];
            } else {
                float* u = u_image<NB>(p, lc, hbase + x2, col / NB) + col % NB;
#pragma unroll
                for (int i = 0; i < kDC; ++i) u[i * (NB + 8)] = x[i];
            }
        }
        __syncthreads();
    }
}

template <int NB>
struct DeltaChainSmem {
    static constexpr int kU = kDC * (NB + 8) * 4;
    static constexpr int kStageW = kDRowsBytes + kDTransBytes + kU + kDVecBytes;               // W | K transposed | U~ | e, D_31
    static constexpr int kStageQ = kDRowsBytes + kDABytes + kDVecBytes;                        // Q | A | e, D_31
    static constexpr int kS = NB * kDLF * 4;                                       // S transposed
    static constexpr int kUb = NB * kDLT * 4;                                      // U transposed
    static constexpr size_t kBytes = static_cast<size_t>(2) * (kStageW + kStageQ + kS + kUb) + kUb + 4 * 8;
};

// Grid (request, head, NB value columns); NB / 2 warps in two halves.  The first half carries the chain: W S, U = U~ - W S, S = e_31 S + K^T (D_31 U),
// with two barriers of its own a chunk.  The second half makes the outputs e Q S + A U beside it, up to a chunk behind: S and U have two
// buffers, `ready` (U of the chunk is there, S was before) and `done` (the outputs have been made) hand them over.  Each half fetches for itself, two
// chunks ahead.  What bounds it is the tensor pipe at the rate of tf32 mma.sync (warps stall on it most) and, next to it, the fragments' splits of
// three instructions a register: 1,511 + 537 tokens, 16 heads 145 us, 5,900 cycles a chunk; with bf16 pairs, split once in memory, 84.
template <int NB>
__global__ void __launch_bounds__(NB * 16, 1)
delta_chain_kernel(const DeltaChunkParams p) {
    pdl_trigger();
    extern __shared__ __align__(128) unsigned char smem[];
    using L = DeltaChainSmem<NB>;
    constexpr int LS = NB + 8, kHalf = NB / 4, kThreads = NB * 16;                 // warps of a half, threads of the block
    unsigned char* sStageW = smem;
    unsigned char* sStageQ = smem + 2 * L::kStageW;
    float* sS = reinterpret_cast<float*>(sStageQ + 2 * L::kStageQ);                // two buffers of S transposed
    float* sU = sS + 2 * NB * kDLF;                                                // two buffers of U transposed
    float* sDU = sU + 2 * NB * kDLT;                                               // D_31 U transposed
    uint64_t* full = reinterpret_cast<uint64_t*>(sDU + NB * kDLT);                 // [2] of the first half, [2] of the second
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int s = blockIdx.x, h = blockIdx.y, cb = blockIdx.z, kvh = h / (p.H / p.G);
    const int slot = p.state_slots[s];
    if (slot < 0 || slot >= p.num_slots) {
        if (threadIdx.x == 0) atomicExch(p.err, 2);
        return;
    }
    int first = 0;                                                                 // the request's first chunk among all
    for (int r = lane; r < s; r += 32) first += chunks_of(p, r);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) first += __shfl_xor_sync(0xffffffffu, first, o);
    const int begin = p.cu_seqlens[s], end = p.cu_seqlens[s + 1];
    const int c0 = max(first, p.c_first), n = min(first + chunks_of(p, s), p.c_first + p.c_count) - c0;      // chunks here
    if (n <= 0) return;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 4; ++i) mbar_init(full + i, 1);
        mbar_fence_init();
    }
    pdl_wait();
    __syncthreads();
    const bool is_q = warp >= kHalf;
    const int w = is_q ? warp - kHalf : warp, m = (w & 1) * 16, nn = (w >> 1) * 8; // the warp's tile of W S or Q S
    auto bulk = [&](unsigned char*& dst, const void* src, int bytes, uint64_t* bar) {
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                     ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
        dst += bytes;
    };
    auto fetch = [&](int c) {                                                      // one thread of a half: chunk c0 + c into the half's stage
        const int st = c & 1, lc = c0 + c - p.c_first;
        const unsigned char* head = head_image(p, lc, h);
        const unsigned char* kv = kv_image(p, lc, kvh);
        uint64_t* bar = full + (is_q ? 2 : 0) + st;
        if (is_q) {
            unsigned char* dst = sStageQ + st * L::kStageQ;
            mbar_expect_tx(bar, L::kStageQ);
            bulk(dst, kv + kDTransBytes, kDRowsBytes, bar);
            bulk(dst, head + kDRowsBytes, kDABytes + kDVecBytes, bar);
        } else {
            unsigned char* dst = sStageW + st * L::kStageW;
            mbar_expect_tx(bar, L::kStageW);
            bulk(dst, head, kDRowsBytes, bar);
            bulk(dst, kv, kDTransBytes, bar);
            bulk(dst, u_image<NB>(p, lc, h, cb), L::kU, bar);
            bulk(dst, head + kDRowsBytes + kDABytes, kDVecBytes, bar);
        }
    };
    if (w == 0 && lane == 0) {
        fetch(0);
        if (n > 1) fetch(1);
    }
    // lhs (32 rows of 128) times the chunk's S: the warp's tile
    auto times_s = [&](float (&a0)[4], const float* lhs, const float* rhs) {
        float x[2][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) { x[i >> 2][i & 3] = 0.f; a0[i & 3] = 0.f; }
        lhs += m * kDLF + a_lane(lane, kDLF);
        rhs += nn * kDLF + b_lane(lane, kDLF);
#pragma unroll
        for (int k = 0; k < kDK / 16; ++k) {
            uint32_t b[4], bh[4], bl[4];
            ldm_x4(b, rhs + k * 16);
            split_tf32(b, bh, bl);
            float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                uint32_t a[4], ah[4], al[4];
                ldm_x4(a, lhs + k * 16 + e * 8);
                split_tf32(a, ah, al);
                mma_1688(c, ah, bh[2 * e], bh[2 * e + 1]);
                mma_1688(x[0], ah, bl[2 * e], bl[2 * e + 1]);
                mma_1688(x[1], al, bh[2 * e], bh[2 * e + 1]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) a0[i] += c[i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) a0[i] += x[0][i] + x[1][i];
    };
    // named barriers: 1 the first half; 2, 3 `ready` and 4, 5 `done` of even and odd chunks
    if (!is_q) {
        // S: four tiles of 16 rows x 8 columns a warp
        auto tile_m = [&](int t) { return (NB == 32 ? w : 2 * w + (t >> 1)) * 16; };
        auto tile_n = [&](int t) { return (NB == 32 ? t : t & 1) * 8; };
        float* st_base = p.state + static_cast<int64_t>(slot) * p.state_floats + static_cast<int64_t>(h) * kDK * p.dv + cb * NB;
        float S[4][4];
        auto write_s = [&](float* dst0) {
#pragma unroll
            for (int t = 0; t < 4; ++t) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    dst0[(tile_n(t) + (lane & 3) * 2 + (e & 1)) * kDLF + tile_m(t) + (lane >> 2) + (e >> 1) * 8] = S[t][e];
            }
        };
#pragma unroll
        for (int t = 0; t < 4; ++t) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const float2 v = *reinterpret_cast<const float2*>(st_base + static_cast<int64_t>(tile_m(t) + (lane >> 2) + half * 8) * p.dv + tile_n(t) + (lane & 3) * 2);
                S[t][half * 2] = v.x;
                S[t][half * 2 + 1] = v.y;
            }
        }
        write_s(sS);
        asm volatile("bar.sync 1, %0;\n" ::"n"(kThreads / 2) : "memory");
        for (int c = 0; c < n; ++c) {
            const int st = c & 1;
            const unsigned char* base = sStageW + st * L::kStageW;
            const float* sW = reinterpret_cast<const float*>(base);
            const float* sKt = reinterpret_cast<const float*>(base + kDRowsBytes);
            const float* sUt = reinterpret_cast<const float*>(base + kDRowsBytes + kDTransBytes);
            const float* sE = sUt + kDC * LS;
            float* u_buf = sU + st * NB * kDLT;
            mbar_wait(full + st, (c >> 1) & 1, p.err);
            float a[4];
            times_s(a, sW, sS + st * NB * kDLF);
#pragma unroll
            for (int half = 0; half < 2; ++half) {                                 // U = U~ - W S, and D_31 U
                const int i = m + (lane >> 2) + half * 8, j = nn + (lane & 3) * 2;
                const float2 ut = *reinterpret_cast<const float2*>(sUt + i * LS + j);
                const float ux = ut.x - a[half * 2], uy = ut.y - a[half * 2 + 1], d = sE[kDC + i];
                sDU[j * kDLT + i] = d * ux;
                sDU[(j + 1) * kDLT + i] = d * uy;
                u_buf[j * kDLT + i] = ux;
                u_buf[(j + 1) * kDLT + i] = uy;
            }
            asm volatile("bar.arrive %0, %1;\n" ::"r"(2 + st), "n"(kThreads) : "memory");        // ready
            asm volatile("bar.sync 1, %0;\n" ::"n"(kThreads / 2) : "memory");
            const float e = sE[kDC - 1];                                           // S = e_31 S + K^T (D_31 U)
            float acc[4][4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[t][i] = 0.f;
            }
            constexpr int kN = NB / 8, kM = 4 / kN;                                // the warp's column and row tiles
#pragma unroll
            for (int k = 0; k < kDC / 16; ++k) {
                uint32_t bh[kN][4], bl[kN][4];
#pragma unroll
                for (int t = 0; t < kN; ++t) {
                    uint32_t b[4];
                    ldm_x4(b, sDU + t * 8 * kDLT + k * 16 + b_lane(lane, kDLT));
                    split_tf32(b, bh[t], bl[t]);
                }
#pragma unroll
                for (int mt = 0; mt < kM; ++mt) {
                    float hh[kN][4], x[kN][4];                                     // a chain of two products, added up by the float units
#pragma unroll
                    for (int i = 0; i < kN * 4; ++i) hh[i >> 2][i & 3] = x[i >> 2][i & 3] = 0.f;
#pragma unroll
                    for (int ee = 0; ee < 2; ++ee) {
                        uint32_t ka[4], kh[4], kl[4];
                        ldm_x4(ka, sKt + tile_m(mt * kN) * kDLT + k * 16 + ee * 8 + a_lane(lane, kDLT));
                        split_tf32(ka, kh, kl);
#pragma unroll
                        for (int t = 0; t < kN; ++t) {
                            mma_1688(hh[t], kh, bh[t][2 * ee], bh[t][2 * ee + 1]);
                            mma_1688(x[t], kh, bl[t][2 * ee], bl[t][2 * ee + 1]);
                            mma_1688(x[t], kl, bh[t][2 * ee], bh[t][2 * ee + 1]);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < kN * 4; ++i) acc[mt * kN + (i >> 2)][i & 3] += hh[i >> 2][i & 3] + x[i >> 2][i & 3];
                }
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
#pragma unroll
                for (int i = 0; i < 4; ++i) S[t][i] = fmaf(e, S[t][i], acc[t][i]);
            }
            if (c > 0) asm volatile("bar.sync %0, %1;\n" ::"r"(4 + (st ^ 1)), "n"(kThreads) : "memory");     // done with the chunk before
            if (c + 1 < n) write_s(sS + (st ^ 1) * NB * kDLF);
            asm volatile("bar.sync 1, %0;\n" ::"n"(kThreads / 2) : "memory");      // the new S is there; the stage may be filled again
            if (threadIdx.x == 0 && c + 2 < n) fetch(c + 2);
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
#pragma unroll
            for (int half = 0; half < 2; ++half)
                *reinterpret_cast<float2*>(st_base + static_cast<int64_t>(tile_m(t) + (lane >> 2) + half * 8) * p.dv + tile_n(t) + (lane & 3) * 2) =
                    make_float2(S[t][half * 2], S[t][half * 2 + 1]);
        }
    } else {
        for (int c = 0; c < n; ++c) {
            const int st = c & 1;
            const float* sQ = reinterpret_cast<const float*>(sStageQ + st * L::kStageQ);
            const float* sA = sQ + kDC * kDLF;
            const float* sE = sA + kDC * kDLT;
            const float* u_buf = sU + st * NB * kDLT;
            mbar_wait(full + 2 + st, (c >> 1) & 1, p.err);
            asm volatile("bar.sync %0, %1;\n" ::"r"(2 + st), "n"(kThreads) : "memory");          // ready
            float o[4];
            times_s(o, sQ, sS + st * NB * kDLF);
            float au[2][4], x[2][4];
#pragma unroll
            for (int i = 0; i < 8; ++i) au[i >> 2][i & 3] = x[i >> 2][i & 3] = 0.f;
#pragma unroll
            for (int k = 0; k < kDC / 16; ++k) {
                uint32_t b[4], bh[4], bl[4];
                ldm_x4(b, u_buf + nn * kDLT + k * 16 + b_lane(lane, kDLT));
                split_tf32(b, bh, bl);
#pragma unroll
                for (int ee = 0; ee < 2; ++ee) {
                    uint32_t ra[4], ah[4], al[4];
                    ldm_x4(ra, sA + m * kDLT + k * 16 + ee * 8 + a_lane(lane, kDLT));
                    split_tf32(ra, ah, al);
                    mma_1688(au[k], ah, bh[2 * ee], bh[2 * ee + 1]);
                    mma_1688(x[0], ah, bl[2 * ee], bl[2 * ee + 1]);
                    mma_1688(x[1], al, bh[2 * ee], bh[2 * ee + 1]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = m + (lane >> 2) + (i >> 1) * 8, col = nn + (lane & 3) * 2 + (i & 1);
                const float qs = o[i] * sE[row];
                o[i] = qs + ((au[0][i] + au[1][i]) + (x[0][i] + x[1][i]));
                // A's zeros above the diagonal times an infinity or a NaN of a later token: the row's own tokens alone, one after the other
                if (!(fabsf(o[i]) <= 3.402823466e38f)) {
                    float own = 0.f;
                    for (int j = 0; j <= row; ++j) own = fmaf(sA[row * kDLT + j], u_buf[col * kDLT + j], own);
                    o[i] = qs + own;
                }
            }
            if (c + 1 < n) asm volatile("bar.arrive %0, %1;\n" ::"r"(4 + st), "n"(kThreads) : "memory");     // done
            const int t0 = begin + (c0 + c - first) * kDC;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int t = t0 + m + (lane >> 2) + half * 8;
                if (t < end)
                    *reinterpret_cast<float2*>(p.out + (static_cast<int64_t>(t) * p.H + h) * p.dv + cb * NB + nn + (lane & 3) * 2) = make_float2(o[half * 2], o[half * 2 + 1]);
            }
            asm volatile("bar.sync 6, %0;\n" ::"n"(kThreads / 2) : "memory");      // the whole half: the stage may be filled again
            if (w == 0 && lane == 0 && c + 2 < n) fetch(c + 2);
        }
    }
}

template <int NB>
int64_t delta_chunk_bytes(int H, int G, int dv) {
    return static_cast<int64_t>(H) * kDHeadBytes + static_cast<int64_t>(G) * kDKvBytes + static_cast<int64_t>(H) * (dv / NB) * kDC * (NB + 8) * 4;
}

template <int NB, int TAPS>
int launch_delta_chunks(DeltaChunkParams p, int total, int held, cudaStream_t stream) {
    static bool set = false;
    if (!set) {
        if (cudaFuncSetAttribute(delta_prepare_kernel<NB, TAPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kDPrepBytes)) != cudaSuccess ||
            cudaFuncSetAttribute(delta_chain_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(DeltaChainSmem<NB>::kBytes)) != cudaSuccess)
            return launch_status();
        set = true;
    }
    // a step of more chunks than the scratch holds goes through it in several turns; the state carries on from one to the next
    for (int c = 0; c < total; c += held) {
        p.c_first = c;
        p.c_count = total - c < held ? total - c : held;
        launch_kernel(delta_prepare_kernel<NB, TAPS>, dim3(p.c_count, p.G), dim3(256), kDPrepBytes, stream, p);
        launch_kernel(delta_chain_kernel<NB>, dim3(p.S, p.H, p.dv / NB), dim3(NB * 16), DeltaChainSmem<NB>::kBytes, stream, p);
    }
    return launch_status();
}

}  // namespace cvb

using namespace cvb;

// Bytes of scratch for `chunks` chunks (of 32 tokens); slices of 16 value columns need the most.
extern "C" int64_t cvb_delta_chunks_scratch(int chunks, int H, int G, int dv) { return static_cast<int64_t>(chunks) * delta_chunk_bytes<16>(H, G, dv); }

// total: the sum over the requests of ceil(tokens / 32).
extern "C" int cvb_delta_chunks(float* out, const void* packed, int stride, int qkv_off, const float* conv_w, int taps, const float* ba,
                                const float* dt_bias, const float* a_log, float* state, int64_t state_floats, int64_t conv_off,
                                const int* cu_seqlens, const int* state_slots, int num_slots, int S, int total, int H, int G, int dk, int dv,
                                void* scratch, int64_t scratch_bytes, int* err_flag, cudaStream_t stream) {
    if (S == 0 || total == 0) return CVB_OK;
    if (S < 0 || total < 0 || H <= 0 || H > 65535 || G <= 0 || num_slots <= 0) return CVB_E_SIZE;
    if (dk != kDK || (dv != 64 && dv != 128) || taps < 1 || taps > 4) return CVB_E_UNSUPPORTED;
    const int64_t C = 2LL * G * dk + static_cast<int64_t>(H) * dv, mat = static_cast<int64_t>(H) * dk * dv;
    if (H % G || qkv_off < 0 || stride < qkv_off + C || conv_off < mat || state_floats < conv_off + (taps - 1) * C) return CVB_E_SHAPE;
    for (const void* p : {static_cast<const void*>(out), static_cast<const void*>(state), static_cast<const void*>(scratch)})
        if (reinterpret_cast<uintptr_t>(p) & 15) return CVB_E_ALIGN;
    // pairs of channels, and a slot's matrices start on whole pairs
    if (state_floats % 2 || stride % 2 || qkv_off % 2 || (reinterpret_cast<uintptr_t>(packed) & 3)) return CVB_E_ALIGN;
    DeltaChunkParams p{};
    p.packed = static_cast<const __nv_bfloat16*>(packed); p.stride = stride; p.qkv_off = qkv_off; p.conv_w = conv_w;
    p.ba = ba; p.dt_bias = dt_bias; p.a_log = a_log; p.conv_off = conv_off;
    p.out = out; p.state = state; p.state_floats = state_floats;
    p.cu_seqlens = cu_seqlens; p.state_slots = state_slots; p.num_slots = num_slots; p.S = S; p.H = H; p.G = G; p.dv = dv;
    p.scratch = static_cast<unsigned char*>(scratch); p.err = err_flag;
    // slices of 16 columns while the chain's blocks fit the SMs at once (each holds an SM's shared memory), else of 32
    const bool narrow = static_cast<int64_t>(S) * H * (dv / 16) <= 148;
    const int64_t per = narrow ? delta_chunk_bytes<16>(H, G, dv) : delta_chunk_bytes<32>(H, G, dv);
    const int64_t fits = scratch_bytes / per;
    if (fits < 1) return CVB_E_SCRATCH;
    const int held = static_cast<int>(fits < total ? fits : total);
#define CALL(T) return narrow ? launch_delta_chunks<16, T>(p, total, held, stream) : launch_delta_chunks<32, T>(p, total, held, stream)
    switch (taps) {
        case 1: CALL(1);
        case 2: CALL(2);
        case 3: CALL(3);
        default: CALL(4);
    }
#undef CALL
}
