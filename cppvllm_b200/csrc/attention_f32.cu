// Attention of prompt portions in true float32 over the paged cache (pages [2][kv head][slot][hd]: keys, then values), causal, with an optional
// window: the arithmetic of attention_general.cu (scale * q.k, online softmax with expf, sum p v / l, all float) by tiles.
//
// attention_general.cu has a block per (token, head): every block reads its keys and values for itself, a thread walks a key's row alone
// (uncoalesced) and a dimension's sum alone.  Here a block owns 64 query rows of one kv head (row r = token r / g, head r % g of the group) and
// walks tiles of 64 keys that arrive by 16-byte cp.async, the next keys while a tile's values are worked on and the other way round.  Two
// halves of 256 threads take every other tile each, with buffers and a running maximum, sum and output of their own, and meet at the end: grids
// are small and one half alone (two warps a scheduler) leaves most latencies in the open.  A half makes S (4 x 4 a thread) and O (4 x hd / 16)
// with register tiles fed by 16-byte shared-memory reads; rows are padded by 4 floats, so that the rows a warp reads side by side fall on
// different banks.  Three prompts of 255, 130 (behind 33) and 64 tokens at 16/8 heads of 128: 433 -> 46 us (one half alone with tiles of 32
// keys 72, both with tiles of 32 keys 51).  Bound by the float units on the SMs with the longest rows (0.58 instructions a cycle there); a finer deal of the rows is left.
#include "common.cuh"
#include "sm100.cuh"

#include <cuda/std/type_traits>

namespace cvb {

constexpr int kFRows = 64;
constexpr int kFKeys = 64;
constexpr int kFPer = kFKeys / 16;                     // keys of S per thread
constexpr int kFThreads = 256;                        // of a half

struct F32AttnParams {
    float* out;                 // [T, H * hd]
    const float* q;             // [T, H * hd]
    const float* pages;         // [num_pages, 2, KV, page_size, hd]
    const int* block_tables;
    const int* cu_seqlens;
    const int* positions;
    int table_width, S, H, KV, page_size, window, num_pages;
    float scale;
    int* err;
};

template <int HD>
struct F32Smem {
    static constexpr int LD = HD + 4;
    static constexpr size_t kBytes = (static_cast<size_t>(kFRows) * LD + 2 * (2 * kFKeys * LD + kFRows * (kFKeys + 4))) * sizeof(float);
};

template <int HD>
__global__ void __launch_bounds__(2 * kFThreads)
attn_prefill_f32_kernel(const F32AttnParams p) {
    pdl_trigger();
    constexpr int LD = HD + 4, LP = kFKeys + 4, CPR = HD / 4;
    extern __shared__ __align__(16) float smf[];
    float* sQ = smf;
    const int part = threadIdx.x / kFThreads;             // which half
    float* sK = sQ + kFRows * LD + part * 2 * kFKeys * LD;                    // the half's keys, then its values
    float* sV = sK + kFKeys * LD;
    float* sP = sQ + kFRows * LD + 2 * 2 * kFKeys * LD + part * kFRows * LP;
    const int tid = threadIdx.x % kFThreads, lane = tid & 31;
    auto half_sync = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(1 + part), "n"(kFThreads) : "memory"); };
    const int g = p.H / p.KV, tok_per_tile = kFRows / g;
    const int kvh = blockIdx.x;
    const int block_id = gridDim.y - 1 - blockIdx.y;      // late blocks (many keys) first
    int seq = -1, q0 = 0, q_len = 0, cu0 = 0, before = 0;
    for (int s0 = 0; s0 < p.S && seq < 0; s0 += 32) {     // the lanes of a warp take a request each (every warp does the same)
        const int s = s0 + lane;
        int a = 0, n = 0;
        if (s < p.S) { a = p.cu_seqlens[s]; n = p.cu_seqlens[s + 1] - a; }
        const int tiles = s < p.S ? (n + tok_per_tile - 1) / tok_per_tile : 0;
        int upto = tiles;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const int first = before + upto - tiles;
        const unsigned hit = __ballot_sync(0xffffffffu, tiles > 0 && block_id >= first && block_id < first + tiles);
        if (hit) {
            const int src = __ffs(hit) - 1;
            seq = s0 + src;
            q0 = (block_id - __shfl_sync(0xffffffffu, first, src)) * tok_per_tile;
            q_len = __shfl_sync(0xffffffffu, n, src);
            cu0 = __shfl_sync(0xffffffffu, a, src);
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (seq < 0) return;
    const int n_tok = min(tok_per_tile, q_len - q0);
    const int* table = p.block_tables + static_cast<int64_t>(seq) * p.table_width;
    const int pos0 = p.positions[cu0 + q0];
    const int key_hi = pos0 + n_tok - 1;                  // a request's tokens of a step sit at consecutive positions
    const int key_lo = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;
    const int last_lo = p.window > 0 ? max(0, key_hi - p.window + 1) : 0;                 // where the last token's window begins
    const int tile0 = key_lo / kFKeys, n_tiles = key_hi / kFKeys - tile0 + 1;
    pdl_wait();
    for (int i = threadIdx.x; i < kFRows * CPR; i += 2 * kFThreads) {
        const int r = i / CPR, c = (i % CPR) * 4, t = r / g;
        const bool valid = t < n_tok;
        const float* src = valid ? p.q + (static_cast<int64_t>(cu0 + q0 + t) * p.H + kvh * g + r - t * g) * HD + c : p.q;
        cp_async16(sQ + r * LD + c, src, valid);
    }
    cp_async_commit();
    auto load_tile = [&](int it, bool values) {           // and a commit
        if (it < n_tiles) {
            float* dst = values ? sV : sK;
            const int key0 = (tile0 + it) * kFKeys;
            for (int i = tid; i < kFKeys * CPR; i += kFThreads) {
                const int r = i / CPR, c = (i % CPR) * 4, j = key0 + r;
                bool need = j <= key_hi && j >= key_lo;   // pages before the window may have been given back
                const float* src = p.pages;
                if (need) {
                    const int slot = j / p.page_size, page = slot < p.table_width ? table[slot] : -1;
                    if (page < 0 || page >= p.num_pages) {
                        atomicExch(p.err, 4);
                        need = false;
                    } else {
                        src = p.pages + (((static_cast<int64_t>(page) * 2 + (values ? 1 : 0)) * p.KV + kvh) * p.page_size + j - slot * p.page_size) * HD + c;
                    }
                }
                cp_async16(dst + r * LD + c, src, need);
            }
        }
        cp_async_commit();
    };
    load_tile(part, false);
    load_tile(part, true);
    // thread (ty, tx): rows ty * 4 .. + 3; of S the keys tx + 16 k; of O the columns tx * 4 + 64 j
    const int ty = tid >> 4, tx = tid & 15;
    int row_pos[4], row_lo[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        row_pos[i] = pos0 + min((ty * 4 + i) / g, n_tok - 1);             // rows past the block's tokens are never stored
        row_lo[i] = p.window > 0 ? max(0, row_pos[i] - p.window + 1) : 0;
    }
    float o[4][HD / 16];
    float m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < HD / 16; ++c) o[i][c] = 0.f;
    }
    cp_async_wait<2>();                                   // the queries, which all threads fetched
    __syncthreads();
    for (int it = part; it < n_tiles; it += 2) {
        cp_async_wait<1>();                               // everything but the newest group, the values: the keys
        half_sync();
        const int key0 = (tile0 + it) * kFKeys;
        float s[4][kFPer];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int k = 0; k < kFPer; ++k) s[i][k] = 0.f;
        }
#pragma unroll 8
        for (int e = 0; e < HD; e += 4) {
            float4 kv[kFPer];
#pragma unroll
            for (int k = 0; k < kFPer; ++k) kv[k] = *reinterpret_cast<const float4*>(sK + (tx + 16 * k) * LD + e);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(sQ + (ty * 4 + i) * LD + e);
#pragma unroll
                for (int k = 0; k < kFPer; ++k) {
                    s[i][k] = fmaf(a.x, kv[k].x, s[i][k]);
                    s[i][k] = fmaf(a.y, kv[k].y, s[i][k]);
                    s[i][k] = fmaf(a.z, kv[k].z, s[i][k]);
                    s[i][k] = fmaf(a.w, kv[k].w, s[i][k]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float top = -INFINITY;
#pragma unroll
            for (int k = 0; k < kFPer; ++k) {
                const int j = key0 + tx + 16 * k;
                s[i][k] = (j <= row_pos[i] && j >= row_lo[i]) ? s[i][k] * p.scale : -INFINITY;
                top = fmaxf(top, s[i][k]);
            }
#pragma unroll
            for (int w = 1; w < 16; w <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, w));
            const float m_new = fmaxf(m[i], top);
            const float corr = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new);
            float sum = 0.f;
#pragma unroll
            for (int k = 0; k < kFPer; ++k) {
                const float pj = s[i][k] == -INFINITY ? 0.f : expf(s[i][k] - m_new);
                sP[(ty * 4 + i) * LP + tx + 16 * k] = pj;
                sum += pj;
            }
#pragma unroll
            for (int w = 1; w < 16; w <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
            l[i] = l[i] * corr + sum;
            m[i] = m_new;
#pragma unroll
            for (int c = 0; c < HD / 16; ++c) o[i][c] *= corr;
        }
        cp_async_wait<0>();
        half_sync();                                      // the values are there, and nobody reads the keys any more
        load_tile(it + 2, false);
        auto weigh = [&](auto edge) {
#pragma unroll 2
            for (int j = 0; j < kFKeys; j += 4) {
                float4 a[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(sP + (ty * 4 + i) * LP + j);
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
#pragma unroll
                    for (int c = 0; c < HD / 64; ++c) {
                        const float4 v = *reinterpret_cast<const float4*>(sV + (j + jj) * LD + c * 64 + tx * 4);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            if (decltype(edge)::value && (key0 + j + jj > row_pos[i] || key0 + j + jj < row_lo[i])) continue;
                            const float pj = jj == 0 ? a[i].x : jj == 1 ? a[i].y : jj == 2 ? a[i].z : a[i].w;
                            o[i][c * 4] = fmaf(pj, v.x, o[i][c * 4]);
                            o[i][c * 4 + 1] = fmaf(pj, v.y, o[i][c * 4 + 1]);
                            o[i][c * 4 + 2] = fmaf(pj, v.z, o[i][c * 4 + 2]);
                            o[i][c * 4 + 3] = fmaf(pj, v.w, o[i][c * 4 + 3]);
                        }
                    }
                }
            }
        };
        // Where some row of the block does not see a key of the tile, that key's value is left out of the row's sum, not weighed with 0: an
        // infinity or a NaN in a later token's value must not reach the tokens before it.
        if (key0 + kFKeys - 1 <= pos0 && key0 >= last_lo) weigh(cuda::std::false_type{});
        else weigh(cuda::std::true_type{});
        half_sync();                                      // nobody reads the values any more
        load_tile(it + 2, true);
    }
    cp_async_wait<0>();
    // the second half leaves its outputs in its keys' and values' room and its maxima and sums in its probabilities', the first one adds them up
    static_assert(2 * kFKeys >= kFRows, "the outputs fit");
    float* const meet = sQ + kFRows * LD + 2 * kFKeys * LD;
    float* const meet_ml = sQ + kFRows * LD + 2 * 2 * kFKeys * LD + kFRows * LP;
    if (part == 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int c = 0; c < HD / 64; ++c)
                *reinterpret_cast<float4*>(meet + (ty * 4 + i) * LD + c * 64 + tx * 4) = make_float4(o[i][c * 4], o[i][c * 4 + 1], o[i][c * 4 + 2], o[i][c * 4 + 3]);
            if (tx == 0) {
                meet_ml[ty * 4 + i] = m[i];
                meet_ml[kFRows + ty * 4 + i] = l[i];
            }
        }
    }
    __syncthreads();
    if (part == 1) return;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float m2 = meet_ml[ty * 4 + i], l2 = meet_ml[kFRows + ty * 4 + i], top = fmaxf(m[i], m2);
        const float f = m[i] == -INFINITY ? 0.f : expf(m[i] - top), f2 = m2 == -INFINITY ? 0.f : expf(m2 - top);
        l[i] = l[i] * f + l2 * f2;
#pragma unroll
        for (int c = 0; c < HD / 64; ++c) {
            const float4 v = *reinterpret_cast<const float4*>(meet + (ty * 4 + i) * LD + c * 64 + tx * 4);
            o[i][c * 4] = o[i][c * 4] * f + v.x * f2;
            o[i][c * 4 + 1] = o[i][c * 4 + 1] * f + v.y * f2;
            o[i][c * 4 + 2] = o[i][c * 4 + 2] * f + v.z * f2;
            o[i][c * 4 + 3] = o[i][c * 4 + 3] * f + v.w * f2;
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i, t = r / g;
        if (t >= n_tok) continue;
        const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
        float* dst = p.out + (static_cast<int64_t>(cu0 + q0 + t) * p.H + kvh * g + r - t * g) * HD + tx * 4;
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
            *reinterpret_cast<float4*>(dst + c * 64) = make_float4(o[i][c * 4] * inv, o[i][c * 4 + 1] * inv, o[i][c * 4 + 2] * inv, o[i][c * 4 + 3] * inv);
    }
}

template <int HD>
int launch_prefill_f32(const F32AttnParams& p, int num_tiles, cudaStream_t stream) {
    static bool set = false;
    if (!set) {
        if (cudaFuncSetAttribute(attn_prefill_f32_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(F32Smem<HD>::kBytes)) != cudaSuccess)
            return launch_status();
        set = true;
    }
    launch_kernel(attn_prefill_f32_kernel<HD>, dim3(p.KV, num_tiles), dim3(2 * kFThreads), F32Smem<HD>::kBytes, stream, p);
    return launch_status();
}

}  // namespace cvb

using namespace cvb;

// num_tiles: per request ceil(tokens / (64 / group)).
extern "C" int cvb_attn_prefill_f32(float* out, const float* q, const float* pages, const int* block_tables, int table_width, const int* cu_seqlens,
                                    const int* positions, int S, int num_tiles, int H, int KV, int hd, int page_size, int window, float scale,
                                    int num_pages, int* err_flag, cudaStream_t stream) {
    if (num_tiles == 0 || S == 0) return CVB_OK;
    if (S < 0 || num_tiles < 0 || num_tiles > 65535 || H <= 0 || KV <= 0 || page_size <= 0 || table_width <= 0 || num_pages <= 0 || window < 0) return CVB_E_SIZE;
    if (H % KV) return CVB_E_SHAPE;
    if ((hd != 64 && hd != 128) || H / KV > kFRows) return CVB_E_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(pages)) & 15) return CVB_E_ALIGN;
    F32AttnParams p{out, q, pages, block_tables, cu_seqlens, positions, table_width, S, H, KV, page_size, window, num_pages, scale, err_flag};
    return hd == 128 ? launch_prefill_f32<128>(p, num_tiles, stream) : launch_prefill_f32<64>(p, num_tiles, stream);
}
