// The state-space recurrence of prompt portions on the fifth-generation tensor cores (tcgen05), in chunks of 128 tokens, for state matrices
// of 128 x 64, at every length (ssd.cu states the recurrence and keeps the other sizes and steps of decoded tokens alone).  Same sums as ssd.cu's:
//   y_t = e^(l_t) S0^T C_t + sum_(s <= t) (C_t . B_s) e^(l_t - l_s) dt_s x_s + D x_t,      S = e^(l_last) S0 + sum_s B_s (e^(l_last - l_s) dt_s x_s)^T
// with the float factors (weights and S0) as two bf16 addends, float accumulation, B, C and x as they are.
//
//   ssd_tc_chunk : per (chunk, group of heads): what the chunk adds to a state from zero.  B is fetched once for the group's heads and is
//                  the transposed operand; two heads at a time, 128 threads each.
//   ssd_tc_carry : the states in front of the chunks, element by element, and the new state.
//   ssd_tc_out   : per (chunk, group of heads): C B^T once, in tensor memory, then head by head: S0's addends through shared memory,
//                  C S0; the scores weighed into tensor memory as two addends, their product with x; y.  The only chunk of a
//                  request (the passes above leave it out) makes the new state.  The next head's S0, x, dt and decays are on their way meanwhile.
// What bounded the chunks of 64 on mma.sync was the states' traffic (a float matrix per chunk and head, written, carried, read: 32 KB for
// 64 tokens) and the fragment loads; chunks of 128 halve the first, and the products read their operands where they lie.  2,048 tokens,
// 32 heads in 8 groups, us (mma.sync in chunks of 64 -> now): chunk pass 21 -> 11.5, carry 13 -> 5.9, outputs 46 -> 19; 128 heads 68 -> 35,
// 53 -> 19.5, 161 -> 64.  What an output block spends on a head (6,500 cycles): S0's addends 620, the next head's fetches 620, weights 1,500, the
// products it cannot hide 650, y 2,000.
// Waits on mbarriers are bounded; one that runs out records error 5 and the block runs on to its end.
#include "common.cuh"
#include "sm100.cuh"

namespace cvb {

constexpr int kTT = 128;                                 // tokens per chunk
constexpr int kTN = 128;                                 // rows of a state
constexpr int kTP = 64;                                  // columns of a state
constexpr int kTThreads = 256;
constexpr int kTTile = kTT * kTP * 2;                    // [128][64] bf16: one 128-byte row per token (or row of S)

struct SsdTcParams {
    float* y;                   // [T, H P]
    const __nv_bfloat16* u;     // rows [x | B | C] of C elements
    const float* dt;            // [T, H]
    const float* la;
    const float* D;             // [H]
    float* ends;
    float* decays;
    float* state;
    int64_t state_floats;
    const int* cu_seqlens;
    const int* state_slots;
    int num_slots, S, H, G, C, heads;      // heads: of a group, per block
    int* err;
};

struct TcChunk { int seq, k, n_chunks, buf, begin, n; };

// Block x's chunk; `buf`: where the request's chunks lie in the chunk buffers, which hold requests with more than one chunk only.  The lanes
// of a warp take a request each (every warp does the same): with a request after the other, 240 decoded tokens beside a portion of 128 made
// a layer of 32 heads take 1,445 us.
__device__ __forceinline__ bool ssd_tc_locate(const SsdTcParams& p, int x, TcChunk& c) {
    const int lane = threadIdx.x & 31;
    int base = 0, held = 0;
    for (int s0 = 0; s0 < p.S; s0 += 32) {
        const int s = s0 + lane;
        int a = 0, tokens = 0;
        if (s < p.S) { a = p.cu_seqlens[s]; tokens = p.cu_seqlens[s + 1] - a; }
        const int chunks = (tokens + kTT - 1) / kTT, many = chunks > 1 ? chunks : 0;
        int upto = chunks, kept = many;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, upto, o), k = __shfl_up_sync(0xffffffffu, kept, o);
            if (lane >= o) { upto += u; kept += k; }
        }
        const int first = base + upto - chunks;
        const unsigned hit = __ballot_sync(0xffffffffu, chunks > 0 && x >= first && x < first + chunks);
        if (hit) {
            const int src = __ffs(hit) - 1;
            c.seq = s0 + src;
            c.k = x - __shfl_sync(0xffffffffu, first, src);
            c.n_chunks = __shfl_sync(0xffffffffu, chunks, src);
            c.buf = held + __shfl_sync(0xffffffffu, kept - many, src);
            c.begin = __shfl_sync(0xffffffffu, a, src) + c.k * kTT;
            c.n = min(kTT, __shfl_sync(0xffffffffu, tokens, src) - c.k * kTT);
            return true;
        }
        base += __shfl_sync(0xffffffffu, upto, 31);
        held += __shfl_sync(0xffffffffu, kept, 31);
    }
    return false;
}

// byte offset of 16-byte chunk c of row r in a tile of 128-byte rows, swizzled
__device__ __forceinline__ int tc_off(int r, int c) { return r * 128 + ((c ^ (r & 7)) << 4); }

// Both halves (64 columns each) of a [128][128] tile of u's columns from `col` on; rows behind the chunk are zeros.
__device__ __forceinline__ void tc_fetch_wide(unsigned char* dst, const SsdTcParams& p, const TcChunk& ck, int col) {
    for (int i = threadIdx.x; i < kTT * 16; i += kTThreads) {
        const int r = i >> 4, c = i & 15;
        const bool in = r < ck.n;
        cp_async16(dst + (c >> 3) * kTTile + tc_off(r, c & 7), in ? p.u + static_cast<int64_t>(ck.begin + r) * p.C + col + c * 8 : p.u, in);
    }
}

// A head's x: [128][64], rows behind the chunk are zeros; by `threads` threads of which this one is t.
__device__ __forceinline__ void tc_fetch_x(unsigned char* dst, const SsdTcParams& p, const TcChunk& ck, int h, int t, int threads) {
    for (int i = t; i < kTT * 8; i += threads) {
        const int r = i >> 3, c = i & 7;
        const bool in = r < ck.n;
        cp_async16(dst + tc_off(r, c), in ? p.u + static_cast<int64_t>(ck.begin + r) * p.C + h * kTP + c * 8 : p.u, in);
    }
}

// Running sums of the decays' logarithms over the 32 tokens of a warp by 128 threads (thread t owns token t), and the four warps' totals; named
// barrier `bar`.  Sums over 32 tokens and not over the chunk: the decay between two tokens is e to a difference of sums, whose rounding
// grows with the sums themselves.  With sums over the chunk, in base 2, y was 1.06 to 1.55 times as far from float64 as that of chunks of 64 with
// decays of e^-0.4 to e^-4 a token on average.
__device__ __forceinline__ float tc_running_sum(float a, float* tot, int t, int bar) {
    const int lane = t & 31, w = t >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, a, o);
        if (lane >= o) a += up;
    }
    if (lane == 31) tot[w] = a;
    asm volatile("bar.sync %0, 128;\n" ::"r"(bar) : "memory");
    return a;
}
// What the 32s from `from` up to `to` (exclusive) add up to; `tot` lies on 16 bytes
__device__ __forceinline__ float tc_between(const float* tot, int from, int to) {
    const float4 v = *reinterpret_cast<const float4*>(tot);
    return ((from <= 0 && to > 0 ? v.x : 0.f) + (from <= 1 && to > 1 ? v.y : 0.f)) + ((from <= 2 && to > 2 ? v.z : 0.f) + (from <= 3 && to > 3 ? v.w : 0.f));
}
// e^d for the decay between two tokens of a 32: 2e-7, and the weight it becomes a factor of keeps 16 bits.  expf here, 32 times a thread and head,
// took 2,048 tokens of 32 heads from 37.3 to 40.6 us and 240 decoded tokens beside a portion from 344 to 395, for the same errors in three digits.
__device__ __forceinline__ float tc_exp(float d) { return ex2(d * 1.4426950408889634f); }
// Logarithm of the decay from a token (running sum l, of 32 number w) to the chunk's end
__device__ __forceinline__ float tc_to_end(const float* tot, int w, float l) { return (tot[w] - l) + tc_between(tot, w + 1, 4); }

// Eight elements of a row of x times w as two bf16 addends, into the rows' tiles hi and lo.
__device__ __forceinline__ void tc_weigh8(unsigned char* hi, unsigned char* lo, int r, int c, uint4 raw, float w) {
    const __nv_bfloat162* x = reinterpret_cast<const __nv_bfloat162*>(&raw);
    uint4 h, l;
    __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&h);
    __nv_bfloat162* l2 = reinterpret_cast<__nv_bfloat162*>(&l);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float2 v = __bfloat1622float2(x[i]);
        v.x *= w; v.y *= w;
        h2[i] = __floats2bfloat162_rn(v.x, v.y);
        const float2 f = __bfloat1622float2(h2[i]);
        l2[i] = __floats2bfloat162_rn(v.x - f.x, v.y - f.y);
    }
    *reinterpret_cast<uint4*>(hi + tc_off(r, c)) = h;
    *reinterpret_cast<uint4*>(lo + tc_off(r, c)) = l;
}

// Instruction descriptors: A K-major or (bit 15) with its rows running, B with its columns running (bit 16) or K-major
constexpr uint32_t kTDescScores = idesc_bf16(kTT, kTT, false);
constexpr uint32_t kTDescCols = idesc_bf16(kTT, kTP, true);
constexpr uint32_t kTDescState = idesc_bf16(kTN, kTP, true) | (1u << 15);

// D += A B of 16 tokens or rows a step with B [128][64] tiles: the low word of a step's descriptor is this much further
constexpr uint32_t kTStep = 16 * 128 >> 4;

// What the chunk adds to a state: columns d .. d + 63 of tensor memory = B^T (hi + lo).  Issued by a whole warp.
__device__ __forceinline__ void tc_issue_state(uint32_t d, const unsigned char* sB, const unsigned char* hi, uint64_t* bar) {
    const uint64_t a = desc_sw128(smem_u32(sB), kTTile, 1024), b = desc_sw128(smem_u32(hi), kTTile, 1024);
    const uint32_t a_lo = static_cast<uint32_t>(a), a_hi = static_cast<uint32_t>(a >> 32), b_lo = static_cast<uint32_t>(b), b_hi = static_cast<uint32_t>(b >> 32);
    if (elect_one()) {
#pragma unroll
        for (int plane = 0; plane < 2; ++plane) {
#pragma unroll
            for (int k = 0; k < kTT / 16; ++k)
                umma(d, desc_words(a_lo + k * kTStep, a_hi), desc_words(b_lo + plane * (kTTile >> 4) + k * kTStep, b_hi), kTDescState, plane + k > 0 ? 1u : 0u);
        }
        tc_commit(bar);
    }
    __syncwarp();
}

constexpr int kTPitch = 272;                             // bytes between rows of a float tile on its way out: 16 pieces and one
constexpr size_t kTChunkSmem = 1024 + 2 * kTTile + 2 * (3 * kTTile + kTN * kTPitch) + 2 * 4 * 4 + 2 * 8 + 16;

// Grid (chunk, group, parts of the group's heads).
__global__ void __launch_bounds__(kTThreads, 1)
ssd_tc_chunk_kernel(const SsdTcParams p) {
    pdl_trigger();
    pdl_wait();
    TcChunk ck;
    if (!ssd_tc_locate(p, blockIdx.x, ck) || ck.n_chunks == 1) return;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* sB = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    unsigned char* planes = sB + 2 * kTTile;             // per pair of heads: hi, lo
    unsigned char* x_tiles = planes + 4 * kTTile;        // per pair of heads: x
    unsigned char* out_tiles = x_tiles + 2 * kTTile;     // per pair of heads: [128][64] float, padded
    float* tot = reinterpret_cast<float*>(out_tiles + 2 * kTN * kTPitch);
    uint64_t* bar = reinterpret_cast<uint64_t*>(tot + 8);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 2);
    const int warp = same_in_warp(threadIdx.x >> 5), part = threadIdx.x >> 7, t = threadIdx.x & 127;
    const int per = p.H / p.G, g = blockIdx.y, h_lo = g * per + blockIdx.z * p.heads, h_hi = min(h_lo + p.heads, (g + 1) * per);
    if (h_lo >= h_hi) return;
    if (threadIdx.x == 0) { mbar_init(bar, 1); mbar_init(bar + 1, 1); mbar_fence_init(); }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(128));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    unsigned char* x_tile = x_tiles + part * kTTile;
    if (h_lo + part < h_hi) tc_fetch_x(x_tile, p, ck, h_lo + part, t, 128);
    cp_async_commit();
    tc_fetch_wide(sB, p, ck, p.H * kTP + g * kTN);
    cp_async_commit();
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = same_in_warp(*tmem_slot);
    unsigned char* hi = planes + part * 2 * kTTile;
    unsigned char* lo = hi + kTTile;
    unsigned char* out_tile = out_tiles + part * kTN * kTPitch;
    for (int h0 = h_lo, round = 0; h0 < h_hi; h0 += 2, ++round) {
        const int h = h0 + part;
        const bool mine = h < h_hi;
        float a = 0.f, d = 0.f;
        if (mine && t < ck.n) {
            a = p.la[static_cast<int64_t>(ck.begin + t) * p.H + h];
            d = p.dt[static_cast<int64_t>(ck.begin + t) * p.H + h];
        }
        if (round == 0) cp_async_wait<1>(); else cp_async_wait<0>();       // x, which the part's threads fetched
        const float l = tc_running_sum(a, tot + part * 4, t, 1 + part);
        const float w = expf(tc_to_end(tot + part * 4, t >> 5, l)) * d;
        if (mine) {
#pragma unroll
            for (int c = 0; c < 8; ++c) tc_weigh8(hi, lo, t, c, *reinterpret_cast<const uint4*>(x_tile + tc_off(t, c)), w);
        }
        if (mine && t == 0) p.decays[static_cast<int64_t>(ck.buf + ck.k) * p.H + h] = expf(tc_between(tot + part * 4, 0, 4));
        cp_async_wait<0>();
        fence_async_smem();
        __syncthreads();
        if (warp == 0) {
            tc_after();
            tc_issue_state(tmem, sB, planes, bar);
            if (h0 + 1 < h_hi) tc_issue_state(tmem + 64, sB, planes + 2 * kTTile, bar + 1);
        }
        if (h + 2 < h_hi) tc_fetch_x(x_tile, p, ck, h + 2, t, 128);
        cp_async_commit();
        if (mine) {
            mbar_wait(bar + part, round & 1, p.err);
            tc_after();
            const uint32_t from = tmem + part * 64 + (static_cast<uint32_t>(warp & 3) << 21);
#pragma unroll
            for (int c0 = 0; c0 < kTP; c0 += 32) {
                uint32_t v[32];
                tm_load32(from + c0, v);
                tm_wait_ld();
#pragma unroll
                for (int c = 0; c < 32; c += 4) *reinterpret_cast<uint4*>(out_tile + t * kTPitch + (c0 + c) * 4) = make_uint4(v[c], v[c + 1], v[c + 2], v[c + 3]);
            }
            tc_before();
            asm volatile("bar.sync %0, 128;\n" ::"r"(1 + part) : "memory");
            const int at = ck.k + 1 < ck.n_chunks ? ck.k + 1 : 0;      // the last chunk's addition waits where the first one's state will lie
            float* dst = p.ends + (static_cast<int64_t>(ck.buf + at) * p.H + h) * (kTN * kTP);
#pragma unroll 8
            for (int i = t; i < kTN * 16; i += 128) *reinterpret_cast<uint4*>(dst + i * 4) = *reinterpret_cast<const uint4*>(out_tile + (i >> 4) * kTPitch + (i & 15) * 16);
        }
    }
    tc_before();
    __syncthreads();
    if (warp == 0) {
        tc_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(128));
    }
}

// ends[buf + k] becomes the state in front of chunk k of every request with more than one chunk.  Grid: (request, head, parts).
__global__ void __launch_bounds__(256)
ssd_tc_carry_kernel(const SsdTcParams p) {
    pdl_trigger();
    pdl_wait();
    const int s = blockIdx.x, h = blockIdx.y;
    const int nc = (p.cu_seqlens[s + 1] - p.cu_seqlens[s] + kTT - 1) / kTT;
    if (nc < 2) return;
    int buf = 0;                                         // the chunks held before the request's
    for (int q = threadIdx.x & 31; q < s; q += 32) {
        const int chunks = (p.cu_seqlens[q + 1] - p.cu_seqlens[q] + kTT - 1) / kTT;
        if (chunks > 1) buf += chunks;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) buf += __shfl_xor_sync(0xffffffffu, buf, o);
    const int slot = p.state_slots[s];
    if (slot < 0 || slot >= p.num_slots) {
        if (threadIdx.x == 0) atomicExch(p.err, 2);
        return;
    }
    constexpr int64_t kMat = kTN * kTP;
    const int64_t step = p.H * kMat, i = (static_cast<int64_t>(blockIdx.z) * 256 + threadIdx.x) * 4;
    float* e0 = p.ends + (static_cast<int64_t>(buf) * p.H + h) * kMat + i;
    const float* d0 = p.decays + static_cast<int64_t>(buf) * p.H + h;
    float* st = p.state + static_cast<int64_t>(slot) * p.state_floats + h * kMat + i;
    const float4 end = *reinterpret_cast<const float4*>(e0);       // what the last chunk adds
    const float a_end = d0[static_cast<int64_t>(nc - 1) * p.H];
    float4 run = *reinterpret_cast<const float4*>(st);
    *reinterpret_cast<float4*>(e0) = run;
    for (int k0 = 1; k0 < nc; k0 += 8) {                 // eight additions on their way at a time
        float4 v[8];
        float a[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (k0 + q < nc) {
                v[q] = *reinterpret_cast<const float4*>(e0 + (k0 + q) * step);
                a[q] = d0[static_cast<int64_t>(k0 + q - 1) * p.H];
            }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (k0 + q < nc) {
                run = make_float4(fmaf(a[q], run.x, v[q].x), fmaf(a[q], run.y, v[q].y), fmaf(a[q], run.z, v[q].z), fmaf(a[q], run.w, v[q].w));
                *reinterpret_cast<float4*>(e0 + (k0 + q) * step) = run;
            }
        }
    }
    *reinterpret_cast<float4*>(st) = make_float4(fmaf(a_end, run.x, end.x), fmaf(a_end, run.y, end.y), fmaf(a_end, run.z, end.z), fmaf(a_end, run.w, end.w));
}

// The scores' part of token t's outputs once more, from the tokens up to t alone: the products weigh later tokens' x with 0, and 0 times
// an infinity is a NaN.
__device__ __noinline__ void tc_own_scores(uint32_t (&q)[32], const unsigned char* sC, const unsigned char* sB, const unsigned char* x_tile,
                                           const float2* ld_h, const float* tot_h, int t, int part) {
    float sum[32];
    for (int c = 0; c < 32; ++c) sum[c] = 0.f;
    for (int s = 0; s <= t; ++s) {
        float score = 0.f;
        for (int c = 0; c < 16; ++c) {
            float a[8], b[8];
            load8(a, reinterpret_cast<const __nv_bfloat16*>(sC + (c >> 3) * kTTile + tc_off(t, c & 7)));
            load8(b, reinterpret_cast<const __nv_bfloat16*>(sB + (c >> 3) * kTTile + tc_off(s, c & 7)));
            for (int k = 0; k < 8; ++k) score = fmaf(a[k], b[k], score);
        }
        const int from = s >> 5, to = t >> 5;
        score *= expf(from == to ? ld_h[t].x - ld_h[s].x : (ld_h[t].x + tc_between(tot_h, from + 1, to)) + (tot_h[from] - ld_h[s].x)) * ld_h[s].y;
        for (int c = 0; c < 4; ++c) {
            float x[8];
            load8(x, reinterpret_cast<const __nv_bfloat16*>(x_tile + tc_off(s, part * 4 + c)));
            for (int k = 0; k < 8; ++k) sum[c * 8 + k] = fmaf(score, x[k], sum[c * 8 + k]);
        }
    }
    for (int c = 0; c < 32; ++c) q[c] = __float_as_uint(sum[c]);
}

constexpr size_t kTOutSmem = 1024 + 8 * kTTile + 2 * kTN * kTP * 4 + 2 * 2 * kTT * 4 + kTT * 4 + 2 * 4 * 4 + 5 * 8 + 16;

// Grid (chunk, group, parts of the group's heads).  Thread (part, t): token t (row t of the state at the end), columns 32 part .. + 31 of y and
// the scores with tokens 64 part .. + 63.  Tensor memory: scores 0..127, their addends 128..191 and 192..255, C S0 (and the state's
// addition) 256..319, scores times x 320..383.
__global__ void __launch_bounds__(kTThreads, 1)
ssd_tc_out_kernel(const SsdTcParams p) {
    pdl_trigger();
    pdl_wait();
    TcChunk ck;
    if (!ssd_tc_locate(p, blockIdx.x, ck)) return;
    const int slot = p.state_slots[ck.seq];
    if (slot < 0 || slot >= p.num_slots) {
        if (threadIdx.x == 0) atomicExch(p.err, 2);
        return;
    }
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* sC = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    unsigned char* sB = sC + 2 * kTTile;
    unsigned char* sS = sB + 2 * kTTile;                 // S0: hi, lo; at the end the weighted rows of x
    unsigned char* sX = sS + 2 * kTTile;                 // this head's x and the next one's
    float* sF = reinterpret_cast<float*>(sX + 2 * kTTile);         // S0 as it arrives
    unsigned char* sY = reinterpret_cast<unsigned char*>(sF + kTN * kTP);                  // y on its way out: [128][64] float, 16-byte pieces swizzled
    float2* ld = reinterpret_cast<float2*>(sY + kTT * kTP * 4);    // [2][128]: running sum over the token's 32, dt
    float* part_w = reinterpret_cast<float*>(ld + 2 * kTT);        // [128]: dt times the decay from a token to the last of its 32
    float* tot = part_w + kTT;                                     // [2][4]: totals of the 32s
    uint64_t* bars = reinterpret_cast<uint64_t*>(tot + 8);         // scores, C S0, scores times x, the state's addition, S0's arrival
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 5);
    const int warp = same_in_warp(threadIdx.x >> 5), part = threadIdx.x >> 7, t = threadIdx.x & 127;
    const int per = p.H / p.G, g = blockIdx.y, h_lo = g * per + blockIdx.z * p.heads, h_hi = min(h_lo + p.heads, (g + 1) * per);
    if (h_lo >= h_hi) return;
    const bool only_chunk = ck.n_chunks == 1;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 5; ++i) mbar_init(bars + i, 1);
        mbar_fence_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    constexpr int64_t kMat = kTN * kTP;
    float* st = p.state + static_cast<int64_t>(slot) * p.state_floats;
    const float* before = ck.n_chunks > 1 ? p.ends + static_cast<int64_t>(ck.buf + ck.k) * p.H * kMat : st;
    float a = 0.f, d = 0.f;
    auto ask = [&](int h, int buf) {                     // a head's state, x, decays and dt; the state's room is free
        if (threadIdx.x == 0) {
            mbar_expect_tx(bars + 4, kMat * 4);
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                         ::"r"(smem_u32(sF)), "l"(before + h * kMat), "r"(static_cast<uint32_t>(kMat * 4)), "r"(smem_u32(bars + 4)) : "memory");
        }
        tc_fetch_x(sX + buf * kTTile, p, ck, h, threadIdx.x, kTThreads);
        if (part == 0) {
            a = t < ck.n ? p.la[static_cast<int64_t>(ck.begin + t) * p.H + h] : 0.f;
            d = t < ck.n ? p.dt[static_cast<int64_t>(ck.begin + t) * p.H + h] : 0.f;
        }
    };
    tc_fetch_wide(sC, p, ck, p.H * kTP + (p.G + g) * kTN);
    tc_fetch_wide(sB, p, ck, p.H * kTP + g * kTN);
    tc_before();
    __syncthreads();
    tc_after();
    ask(h_lo, 0);
    cp_async_commit();
    const uint32_t tmem = same_in_warp(*tmem_slot), lanes = static_cast<uint32_t>(warp & 3) << 21;
    const uint64_t k_desc = desc_sw128(smem_u32(sC), 16, 1024), mn_desc = desc_sw128(smem_u32(sS), kTTile, 1024);
    const uint32_t c_lo = static_cast<uint32_t>(k_desc), k_hi = static_cast<uint32_t>(k_desc >> 32), b_lo = c_lo + (2 * kTTile >> 4);
    const uint32_t s_lo = static_cast<uint32_t>(mn_desc), mn_hi = static_cast<uint32_t>(mn_desc >> 32), x_lo = s_lo + (2 * kTTile >> 4);
    auto k_step = [](int k) { return (k >> 2) * (kTTile >> 4) + (k & 3) * 2; };             // 16 of K further in a K-major [128][128] tile
    for (int h = h_lo, i = 0; h < h_hi; ++h, ++i) {
        const int buf = i & 1;
        unsigned char* x_tile = sX + buf * kTTile;
        float2* ld_h = ld + buf * kTT;
        float* tot_h = tot + buf * 4;
        if (part == 0) {
            const float l = tc_running_sum(a, tot_h, t, 1);
            ld_h[t] = make_float2(l, d);
            part_w[t] = expf(__shfl_sync(0xffffffffu, l, 31) - l) * d;
        }
        mbar_wait(bars + 4, i & 1, p.err);
#pragma unroll
        for (int j = 0; j < 8; ++j) {                    // S0 as two addends
            const int idx = threadIdx.x + j * kTThreads, r = idx >> 4, c4 = idx & 15;
            const float4 v = *reinterpret_cast<const float4*>(sF + idx * 4);
            const __nv_bfloat162 h0 = __floats2bfloat162_rn(v.x, v.y), h1 = __floats2bfloat162_rn(v.z, v.w);
            const float2 f0 = __bfloat1622float2(h0), f1 = __bfloat1622float2(h1);
            const __nv_bfloat162 l0 = __floats2bfloat162_rn(v.x - f0.x, v.y - f0.y), l1 = __floats2bfloat162_rn(v.z - f1.x, v.w - f1.y);
            unsigned char* at = sS + tc_off(r, c4 >> 1) + (c4 & 1) * 8;
            *reinterpret_cast<uint2*>(at) = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
            *reinterpret_cast<uint2*>(at + kTTile) = make_uint2(*reinterpret_cast<const uint32_t*>(&l0), *reinterpret_cast<const uint32_t*>(&l1));
        }
        cp_async_wait<0>();
        fence_async_smem();
        tc_before();
        __syncthreads();
        tc_after();
        if (warp == 0) {
            if (elect_one()) {
                if (i == 0) {                            // C B^T, for all heads of the group
#pragma unroll
                    for (int k = 0; k < kTN / 16; ++k)
                        umma(tmem, desc_words(c_lo + k_step(k), k_hi), desc_words(b_lo + k_step(k), k_hi), kTDescScores, k > 0 ? 1u : 0u);
                    tc_commit(bars);
                }
#pragma unroll
                for (int plane = 0; plane < 2; ++plane) {
#pragma unroll
                    for (int k = 0; k < kTN / 16; ++k)
                        umma(tmem + 256, desc_words(c_lo + k_step(k), k_hi), desc_words(s_lo + plane * (kTTile >> 4) + k * kTStep, mn_hi), kTDescCols,
                             plane + k > 0 ? 1u : 0u);
                }
                tc_commit(bars + 1);
            }
            __syncwarp();
        }
        if (h + 1 < h_hi) ask(h + 1, buf ^ 1);
        cp_async_commit();
        if (i == 0) { mbar_wait(bars, 0, p.err); tc_after(); }
        const float l_t = ld_h[t].x;                     // over the token's 32
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {           // tokens s by 32; the parts take every other 32
            const int block = half * 2 + part, first = block * 32, own = warp & 3;
            uint32_t hi[16], lo[16];
            if (block <= own) {                          // the warp's tokens see some of them
                uint32_t v[32];
                tm_load32(tmem + lanes + first, v);
                tm_wait_ld();
                auto put = [&](int k, float2 e) {
                    const __nv_bfloat162 h2 = __floats2bfloat162_rn(e.x, e.y);
                    const float2 f = __bfloat1622float2(h2);
                    const __nv_bfloat162 l2 = __floats2bfloat162_rn(e.x - f.x, e.y - f.y);
                    hi[k] = *reinterpret_cast<const uint32_t*>(&h2);
                    lo[k] = *reinterpret_cast<const uint32_t*>(&l2);
                };
                if (block < own) {                       // all of them: the decay is that to the 32's last token and that from there on, neither above 1
                    const float on = expf(l_t + tc_between(tot_h, block + 1, own));
                    const float2 on2 = make_float2(on, on);
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        const float2 w = *reinterpret_cast<const float2*>(part_w + first + 2 * k);
                        put(k, __fmul2_rn(make_float2(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1])), __fmul2_rn(w, on2)));
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        const float4 w = *reinterpret_cast<const float4*>(ld_h + first + 2 * k);           // l, dt of two neighbours
                        put(k, make_float2(first + 2 * k <= t ? __uint_as_float(v[2 * k]) * tc_exp(l_t - w.x) * w.y : 0.f,
                                           first + 2 * k + 1 <= t ? __uint_as_float(v[2 * k + 1]) * tc_exp(l_t - w.z) * w.w : 0.f));
                    }
                }
            } else {
#pragma unroll
                for (int k = 0; k < 16; ++k) hi[k] = lo[k] = 0u;
            }
            tm_store16(tmem + lanes + 128 + first / 2, hi);
            tm_store16(tmem + lanes + 192 + first / 2, lo);
        }
        tm_wait_st();
        tc_before();
        __syncthreads();
        tc_after();
        if (warp == 0) {
            const uint32_t xl = x_lo + buf * (kTTile >> 4);
            if (elect_one()) {
#pragma unroll
                for (int plane = 0; plane < 2; ++plane) {
#pragma unroll
                    for (int k = 0; k < kTT / 16; ++k)
                        umma_ts(tmem + 320, tmem + 128 + plane * 64 + k * 8, desc_words(xl + k * kTStep, mn_hi), kTDescCols, plane + k > 0 ? 1u : 0u);
                }
                tc_commit(bars + 2);
            }
            __syncwarp();
        }
        const float skip = p.D[h], grow = expf(tc_between(tot_h, 0, t >> 5) + l_t);
        mbar_wait(bars + 1, i & 1, p.err);
        mbar_wait(bars + 2, i & 1, p.err);
        tc_after();
        uint32_t o[32], q[32];
        tm_load32(tmem + lanes + 256 + part * 32, o);
        tm_load32(tmem + lanes + 320 + part * 32, q);
        tm_wait_ld();
        bool bad = false;
#pragma unroll
        for (int c = 0; c < 32; ++c) bad = bad || !(fabsf(__uint_as_float(q[c])) <= 3.402823466e38f);
        if (bad) tc_own_scores(q, sC, sB, x_tile, ld_h, tot_h, t, part);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float x[8];
            load8(x, reinterpret_cast<const __nv_bfloat16*>(x_tile + tc_off(t, part * 4 + c)));
            float r[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) r[k] = fmaf(skip, x[k], fmaf(grow, __uint_as_float(o[c * 8 + k]), __uint_as_float(q[c * 8 + k])));
#pragma unroll
            for (int k = 0; k < 2; ++k)
                *reinterpret_cast<float4*>(sY + t * 256 + (((part * 8 + c * 2 + k) ^ (t & 7)) << 4)) = make_float4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
        }
        __syncthreads();
        for (int j = threadIdx.x; j < ck.n * 16; j += kTThreads) {
            const int r = j >> 4, c = j & 15;
            *reinterpret_cast<float4*>(p.y + (static_cast<int64_t>(ck.begin + r) * p.H + h) * kTP + c * 4) = *reinterpret_cast<const float4*>(sY + r * 256 + ((c ^ (r & 7)) << 4));
        }
        if (only_chunk) {                                // the request's new state
            const float w = expf(tc_to_end(tot_h, t >> 5, l_t)) * ld_h[t].y, keep = expf(tc_between(tot_h, 0, 4));
            float* at = st + h * kMat;
            float4 old[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) old[j] = *reinterpret_cast<const float4*>(at + (threadIdx.x + j * kTThreads) * 4);
#pragma unroll
            for (int c = 0; c < 4; ++c) tc_weigh8(sS, sS + kTTile, t, part * 4 + c, *reinterpret_cast<const uint4*>(x_tile + tc_off(t, part * 4 + c)), w);
            fence_async_smem();
            tc_before();
            __syncthreads();
            tc_after();
            if (warp == 0) tc_issue_state(tmem + 256, sB, sS, bars + 3);
            mbar_wait(bars + 3, i & 1, p.err);
            tc_after();
            tm_load32(tmem + lanes + 256 + part * 32, o);
            tm_wait_ld();
#pragma unroll
            for (int c = 0; c < 8; ++c)
                *reinterpret_cast<uint4*>(sY + t * 256 + (((part * 8 + c) ^ (t & 7)) << 4)) = make_uint4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
            __syncthreads();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int idx = threadIdx.x + j * kTThreads, r = idx >> 4, c = idx & 15;
                const float4 v = *reinterpret_cast<const float4*>(sY + r * 256 + ((c ^ (r & 7)) << 4));
                *reinterpret_cast<float4*>(at + idx * 4) = make_float4(fmaf(keep, old[j].x, v.x), fmaf(keep, old[j].y, v.y), fmaf(keep, old[j].z, v.z), fmaf(keep, old[j].w, v.w));
            }
        }
    }
    tc_before();
    __syncthreads();
    if (warp == 0) {
        tc_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
    }
}

}  // namespace cvb

using namespace cvb;

// `chunks`: how many chunks of 128 tokens the step's requests have together; `held`: how many of them belong to requests with more than
// one (0: the outputs' pass alone runs); `ends` holds H * 128 * 64 floats and `decays` H floats per held chunk.  u: bf16 rows [x | B | C].
extern "C" int cvb_ssd_chunks_tcgen05(float* y, const void* u, const float* dt, const float* la, const float* D, float* ends, int64_t ends_floats,
                                      float* decays, int64_t decays_floats, float* state, int64_t state_floats, int num_slots, const int* cu_seqlens,
                                      const int* state_slots, int S, int chunks, int held, int H, int G, int N, int P, int* err_flag,
                                      cudaStream_t stream) {
    if (S == 0) return CVB_OK;
    if (S < 0 || chunks <= 0 || held < 0 || H <= 0 || G <= 0 || num_slots <= 0 || H > 65535 || G > 65535) return CVB_E_SIZE;
    if (H % G) return CVB_E_SHAPE;
    if (N != kTN || P != kTP) return CVB_E_UNSUPPORTED;
    const int64_t C = static_cast<int64_t>(H) * P + 2LL * G * N, mat = static_cast<int64_t>(N) * P;
    if (state_floats < H * mat || C > 2147483647LL) return CVB_E_SHAPE;
    auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    if (!al(u) || !al(y) || !al(state) || state_floats % 4 || (held > 0 && !al(ends))) return CVB_E_ALIGN;
    if (held > 0 && (ends == nullptr || decays == nullptr || ends_floats < held * H * mat || decays_floats < static_cast<int64_t>(held) * H)) return CVB_E_SCRATCH;
    static bool raised = false;
    if (!raised) {
        if (cudaFuncSetAttribute(ssd_tc_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTChunkSmem)) != cudaSuccess ||
            cudaFuncSetAttribute(ssd_tc_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTOutSmem)) != cudaSuccess)
            return launch_status();
        raised = true;
    }
    SsdTcParams p{y, static_cast<const __nv_bfloat16*>(u), dt, la, D, ends, decays, state, state_floats, cu_seqlens, state_slots, num_slots, S, H, G,
                  static_cast<int>(C), 0, err_flag};
    // a group's heads stay together (they share B, C and C B^T) while the blocks fill the SMs, else they are dealt out
    const int per = H / G;
    int64_t parts = 148 / (static_cast<int64_t>(chunks) * G);
    parts = parts < 1 ? 1 : (parts > per ? per : parts);
    p.heads = static_cast<int>((per + parts - 1) / parts);
    const unsigned pz = static_cast<unsigned>((per + p.heads - 1) / p.heads);
    if (held > 0) {
        launch_kernel(ssd_tc_chunk_kernel, dim3(chunks, G, pz), dim3(kTThreads), kTChunkSmem, stream, p);
        launch_kernel(ssd_tc_carry_kernel, dim3(S, H, kTN * kTP / 1024), dim3(256), 0, stream, p);
    }
    launch_kernel(ssd_tc_out_kernel, dim3(chunks, G, pz), dim3(kTThreads), kTOutSmem, stream, p);
    return launch_status();
}
