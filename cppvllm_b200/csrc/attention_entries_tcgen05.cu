// Attention of prompt portions on the fifth-generation tensor cores (tcgen05), bf16, over pages of cache entries: a key and, behind
// it, its value ([plane][kv head][slot][dk + dv]; attention_masked.cu and attention_bias.cu state the masks and score terms), or keys
// whose leading elements are the values ([kv head][slot][HD]; attention_keys.cu).  Sizes: keys of 64 or 128 elements, values as wide
// (of a shared entry also 96 of 128), pages of 16 tokens or more.  Same arithmetic as those files' mma.sync kernels, which keep the
// other sizes: scores, maxima, sums and output in float, probabilities rounded to bf16 for the product with the values.
//
// What bounds the mma.sync kernels is the legacy tensor path and the shared-memory reads that feed it: 64 query rows per block and
// 64 keys per tile, every operand fragment through ldmatrix.  Here a block owns 256 query rows of one kv head as two tiles of 128 (row r
// of a tile = token r / g, head r % g of the group), walks tiles of 128 entries, and the tensor core alternates between the two query
// tiles, as in attention_tcgen05.cu.  Measured, 2,048 tokens at 16/8 heads of 128 (us, mma.sync -> now): chunks of 1,024 179 -> 27; a latent of
// 96 + 32 under 16 heads 171 -> 39; a bias per distance (1,500 tokens and 548 behind 700) 211 -> 40; keys that are values at 32/8 heads
// (1,917 tokens of three requests behind a window of 1,024) 196 -> 43.
//   warp 0     producer: one lane per TMA box (page or 64 entries, times 64 columns, times key and value), 128-byte swizzle.  Key and
//              value apart: two stages, each with the keys of tile i + 1 and the values of tile i (what one round reads).  Shared
//              entries: four stages of one tile, read row-wise by S = Q K^T and transposed by O += P K;
//   warp 1     allocates 512 columns of tensor memory and issues the products: P_i V_i in two halves as P is handed over, then S_{i+1},
//              for either query tile; the whole warp walks the list with values that are the same in all lanes and one lane issues (the
//              four cases above: 29.5, 44.6, 48.1, 50.8 from one thread's branch, 28.7, 42.3, 44.6, 47.5 so);
//   warps 4-11 softmax, one thread per query row: S from tensor memory, scale, cap, term by distance, mask, exponentials, P back over
//              S; O is rescaled in tensor memory when some row of the warp has a new maximum.  The reference is the maximum itself, so that a row's
//              largest probability is 1 and rounds to 1: with one that followed only after 2^8, layers were 1 to 5 % further from float64 (capped
//              scores 4.00e-3 -> 4.22e-3, a bias per distance 4.82e-3 -> 4.90e-3) and 2 to 5 % faster (a bias per distance 79 us against 83).
//              All exponentials are the special-function unit's (a third of them as a polynomial on the multiply-add units: 25.5, 36.0,
//              -, 40.8 us where 26.8, 39.1, 39.9, 42.7, and coarser: attention_tcgen05.cu).
// The tiles a block walks are a list: pooled blocks any of its tokens sees (plane 1), kept first tokens that lie wholly before the
// rest, then the tokens from the first one its first token sees to its last token; a query tile skips list entries it sees nothing of.
//   distance terms: bias[h, min(p - j, L - 1)] or -r1_h ln(1 + r2_h (p - j)) come from a table in shared memory, one row per head of
//       the group, in log2 units, padded at both ends so that a thread reads 128 neighbours at immediate offsets (rows of
//       neighbouring heads start 32 / g banks apart: no conflicts for g = 2^n);
//   cap: c tanh(s / c) by an odd polynomial up to x^11 where the warp's scores stay below 0.4 c (error below 3e-8, what the
//       exponential form has), by the exponential form elsewhere: two MUFU operations an element less where they are the bound.
// Entries of a tile that no token of the block sees are zeroed in shared memory before the product with P reads them (a stale page
// may hold anything, and 0 times an Inf is a NaN).  A grid with few query blocks of many tiles each leaves SMs idle, so the tiles of a
// query block may be shared out among up to eight blocks ("pieces"); they leave unnormalised rows, maxima and sums in scratch and
// attn_entries_merge_kernel adds them up.  Waits are bounded; one that runs out records error 5 and the block runs on to its end.
#include "sm100.cuh"
#include "tensor_map.cuh"

namespace cvb {

constexpr int kEM = 128;                      // query rows per tile
constexpr int kEN = 128;                      // entries per tile
constexpr int kEThreads = 128 + 256;          // one warpgroup of helpers (two warps idle), one warpgroup per query tile
constexpr float kELog2e = 1.4426950408889634f;
constexpr int kEMaxPieces = 8;
constexpr int kEPadHigh = 160;                // entries behind a distance table's last one: 127 keys and 32 tokens of a warp

// element offset of 16-byte chunk c of row r in a [128 rows][HD] tile stored as HD/64 halves of [128][64], swizzled
__device__ __forceinline__ int entry_off(int r, int c) { return ((c >> 3) << 13) + (r << 6) + (((c & 7) ^ (r & 7)) << 3); }

struct EntryAttnParams {
    __nv_bfloat16* out;                 // rows of out_stride elements, H * DV of them used
    const __nv_bfloat16* q;             // rows of q_stride elements, the first H * HD the queries
    const __nv_bfloat16* gate;          // rows of gate_stride elements or null: a column per head, or (gate_element) per element
    const float* bias;                  // [H, bias_len] or null
    const float* r1;                    // [H] or null
    const float* r2;
    const float* sink;                  // [H] or null
    const int* block_tables;
    const int* cu_seqlens;
    const int* positions;
    int q_stride, out_stride, gate_stride, gate_element;
    int table_width, S, H, G, page_size, planes, num_pages, box_rows;
    int chunk, window, pool, keep;
    int table_len, table_stride;        // distance table in shared memory: entries without the pads (0: none), floats per head
    int bias_len;
    float scale, softcap, out_scale;
    int* err;
    int pieces, min_rounds;
    float* part_o;                      // [query block * kv head * pieces][2 query tiles][DV][128 rows]
    float* part_ml;                     // [query block * kv head * pieces][2 query tiles][maximum | sum][128 rows]
    int* piece_counts;                  // [query block * kv head]: into how many pieces the block was cut (written by piece 0)
};

__device__ __forceinline__ int entry_first_visible(int p, const EntryAttnParams& a) {
    int lo = 0;
    if (a.chunk > 0) lo = p / a.chunk * a.chunk;
    if (a.window > 0) lo = max(lo, p - a.window + 1);
    return lo;
}
__device__ __forceinline__ int entry_visible_blocks(int p, const EntryAttnParams& a) {
    return (a.pool > 0 && a.window > 0) ? max(0, (p - a.window + 1) / a.pool) : 0;
}

// Which request query block `block_id` belongs to: the lanes of a warp take a request each, count its query blocks, add them up with
// shuffles and see whose range holds block_id.
__device__ __forceinline__ int entry_find_block(const EntryAttnParams& p, int block_id, int tok_per_block, int lane, int& q0, int& q_len, int& cu0) {
    int seq = -1, before = 0;
    for (int s0 = 0; s0 < p.S && seq < 0; s0 += 32) {
        const int s = s0 + lane;
        int a = 0, n = 0;
        if (s < p.S) { a = p.cu_seqlens[s]; n = p.cu_seqlens[s + 1] - a; }
        const int tiles = s < p.S ? (n + tok_per_block - 1) / tok_per_block : 0;
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
            q0 = (block_id - __shfl_sync(0xffffffffu, first, src)) * tok_per_block;
            q_len = __shfl_sync(0xffffffffu, n, src);
            cu0 = __shfl_sync(0xffffffffu, a, src);
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    return seq;
}

template <int HD>
struct EntrySmem {
    static constexpr int kTile = 128 * HD * 2;
    static constexpr int kNumBars = 4 + 4 + 2 + 4 + 2;
    static constexpr size_t kBytes = static_cast<size_t>(kTile) * 6 + kNumBars * 8 + 16;      // and the distance table behind it
};

// tanh(x) for |x| <= 0.4: the odd Taylor series up to x^11 (the next term is below 2.5e-8 there), two at a time
__device__ __forceinline__ float2 tanh_small2(float2 x) {
    const float2 y = __fmul2_rn(x, x);
    float2 t = make_float2(-1382.f / 155925.f, -1382.f / 155925.f);
    t = __ffma2_rn(t, y, make_float2(62.f / 2835.f, 62.f / 2835.f));
    t = __ffma2_rn(t, y, make_float2(-17.f / 315.f, -17.f / 315.f));
    t = __ffma2_rn(t, y, make_float2(2.f / 15.f, 2.f / 15.f));
    t = __ffma2_rn(t, y, make_float2(-1.f / 3.f, -1.f / 3.f));
    t = __ffma2_rn(t, y, make_float2(1.f, 1.f));
    return __fmul2_rn(t, x);
}
__device__ __forceinline__ float tanh_exponential(float x) { return 1.f - __fdividef(2.f, 1.f + __expf(2.f * x)); }

// SHARED: one entry is key and value.  TERMS: a cap or a distance table (else the scale joins the exponent's multiply-add, behind the mask and
// the maximum: it must be above 0).
template <int HD, int DV, bool SHARED, bool TERMS>
__global__ void __launch_bounds__(kEThreads, 1)
attn_entries_tcgen05_kernel(const __grid_constant__ CUtensorMap map, const EntryAttnParams p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    using L = EntrySmem<HD>;
    constexpr int kStages = SHARED ? 4 : 2;
    constexpr int kLag = SHARED ? 0 : 1;          // load i brings the keys of tile i and the values of tile i - kLag
    pdl_trigger();
    if ((smem_u32(smem_raw) & 1023u) != 0) {
        if (threadIdx.x == 0) atomicExch(p.err, 6);
        return;
    }
    unsigned char* sQ = smem_raw;                                   // two tiles
    unsigned char* sKV = sQ + 2 * L::kTile;                         // stage s: keys at (2 s), values at (2 s + 1); shared: entries at s
    uint64_t* bars = reinterpret_cast<uint64_t*>(sKV + 4 * L::kTile);
    uint64_t* kv_full = bars;                      // TMA: what the stage holds has landed
    uint64_t* kv_empty = kv_full + 4;              // tensor core: the products that read the stage are done
    uint64_t* s_ready = kv_empty + 4;              // [2 query tiles]  tensor core: S(X) and everything issued before it is done
    uint64_t* p_ready = s_ready + 2;               // [2 query tiles][2 halves of the tile's entries]  128 softmax threads: P(X) is in tensor memory
    uint64_t* o_done = p_ready + 4;                // [2 query tiles]  tensor core: the last PV(X) is done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);
    float* sT = reinterpret_cast<float*>(tmem_slot + 4);            // distance table [g][table_stride]

    const int warp = same_in_warp(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int g = p.H / p.G;
    const int tok_per_tile = kEM / g;
    const int tok_per_block = 2 * tok_per_tile;
    const int kvh = blockIdx.x;
    constexpr int CPR = HD / 8;

    // Blocks are handed out with the kv head running fastest, then the query block, late ones (long lists) first, then the piece.
    const int block_id = gridDim.y - 1 - blockIdx.y, piece = blockIdx.z;
    int q0 = 0, q_len = 0, cu0 = 0;
    const int seq = entry_find_block(p, block_id, tok_per_block, lane, q0, q_len, cu0);
    if (seq < 0) return;
    const int* table = p.block_tables + static_cast<int64_t>(seq) * p.table_width;
    int n_tok[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) n_tok[x] = max(0, min(tok_per_tile, q_len - q0 - x * tok_per_tile));
    // r / g for r < 256 without a division (g <= 128): checked for every pair by a test on the host
    const uint32_t g_mul = ((1u << 20) + g - 1) / g;
    auto row_tok = [&](int r) { return static_cast<int>((static_cast<uint32_t>(r) * g_mul) >> 20); };
    // positions are a step input, in place before the first kernel of the step: read ahead of griddepcontrol.wait.  A request's
    // tokens of a step sit at consecutive positions.
    const int pos0 = p.positions[cu0 + q0];
    const int first_pos[2] = {pos0, pos0 + tok_per_tile};
    const int last_pos[2] = {pos0 + n_tok[0] - 1, pos0 + tok_per_tile + n_tok[1] - 1};
    const int key_hi = pos0 + n_tok[0] + n_tok[1] - 1;              // the block's last token

    // the list of tiles
    const int nb_max = entry_visible_blocks(key_hi, p);
    const int n_pool = (nb_max + kEN - 1) / kEN;
    const int key_lo = entry_first_visible(pos0, p), keep = p.window > 0 ? p.keep : 0;
    const int tok0 = key_lo / kEN;
    const int n_kept = keep > 0 ? min((keep - 1) / kEN + 1, tok0) : 0;
    const int n_list = n_pool + n_kept + key_hi / kEN - tok0 + 1;
    auto first_key = [&](int it) {
        if (it < n_pool) return it * kEN;
        it -= n_pool;
        return (it < n_kept ? it : tok0 + it - n_kept) * kEN;
    };
    const int lo_b = entry_first_visible(first_pos[1], p), nb_a = entry_visible_blocks(last_pos[0], p);
    auto active = [&](int x, int it) {
        const int key0 = first_key(it);
        if ((x ? n_tok[1] : n_tok[0]) == 0) return false;
        if (it < n_pool) return key0 < (x ? nb_max : nb_a);
        return key0 <= (x ? last_pos[1] : last_pos[0]) && (key0 + kEN > (x ? lo_b : key_lo) || key0 < keep);
    };
    int it_lo = 0, it_hi = n_list, n_pieces = 1;
    if (p.pieces > 1) {
        n_pieces = min(p.pieces, max(1, n_list / p.min_rounds));
        if (piece >= n_pieces) return;
        it_lo = n_list * piece / n_pieces;
        it_hi = n_list * (piece + 1) / n_pieces;
    }
    int last_it[2];                                                 // the query tile's last list entry here, or -1
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        int it = it_hi - 1;
        while (it >= it_lo && !active(x, it)) --it;
        last_it[x] = it >= it_lo ? it : -1;
    }
    const int part_slot = (block_id * p.G + kvh) * p.pieces + piece;
    pdl_wait();
    if (p.pieces > 1 && piece == 0 && threadIdx.x == 0) p.piece_counts[block_id * p.G + kvh] = n_pieces;

    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < 4; ++i) { mbar_init(kv_full + i, 1); mbar_init(kv_empty + i, 1); }
            for (int i = 0; i < 2; ++i) { mbar_init(s_ready + i, 1); mbar_init(o_done + i, 1); }
            for (int i = 0; i < 4; ++i) mbar_init(p_ready + i, 128);
            mbar_fence_init();
        }
        __syncwarp();
        asm volatile("bar.arrive 1, %0;\n" ::"n"(kEThreads) : "memory");       // the others wait for this below
    } else {
        if (warp == 1) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(512));
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
        }
        // query rows: row r of tile x = (token x * tok_per_tile + r / g, head kvh * g + r % g); rows past the portion are zero
        const __nv_bfloat16* q_base = p.q + static_cast<int64_t>(cu0 + q0) * p.q_stride + kvh * g * HD;
        for (int i = threadIdx.x - 32; i < 2 * kEM * CPR; i += kEThreads - 32) {
            const int row = i / CPR, c = i % CPR;
            const int x = row >> 7, r = row & 127;
            const int t = row_tok(r), h = r - t * g;
            const bool valid = t < n_tok[x];
            const __nv_bfloat16* src = valid ? q_base + static_cast<int64_t>(x * tok_per_tile + t) * p.q_stride + h * HD + c * 8 : p.q;
            cp_async16(reinterpret_cast<__nv_bfloat16*>(sQ + x * L::kTile) + entry_off(r, c), src, valid);
        }
        cp_async_commit();
        if (TERMS && p.table_len > 0) {
            // row h: tok_per_tile + 128 entries for distances below 0 (masked scores), the distances, kEPadHigh times the last one; as
            // far as the block's entries reach
            const int pad = tok_per_tile + kEN, reach = key_hi - (keep > 0 ? 0 : tok0 * kEN) + 1;
            const int len = pad + (reach < p.table_len ? reach : p.table_len + kEPadHigh);
            for (int idx = threadIdx.x - 32; idx < g * len; idx += kEThreads - 32) {
                const int h = idx / len, i = idx - h * len, head = kvh * g + h;
                const int d = min(max(i - pad, 0), p.table_len - 1);
                float v = 0.f;
                if (p.bias != nullptr) v = p.bias[static_cast<int64_t>(head) * p.bias_len + d];
                if (p.r1 != nullptr) v -= p.r1[head] * __logf(1.f + p.r2[head] * static_cast<float>(d));
                sT[h * p.table_stride + i] = v * kELog2e;
            }
        }
        cp_async_wait<0>();
        fence_async_smem();                                         // the tensor core reads what these threads wrote
        tc_before();
        asm volatile("bar.sync 1, %0;\n" ::"n"(kEThreads) : "memory");
        tc_after();
    }
    const uint32_t tmem = warp == 0 ? 0u : *tmem_slot;
    const uint32_t tS[2] = {tmem, tmem + 128};
    const uint32_t tO[2] = {tmem + 256, tmem + 256 + HD};
    auto entry_tile = [&](int i, bool value) {                      // where list entry it_lo + i lies, as key or as value
        if (SHARED) return sKV + (i % kStages) * L::kTile;
        return sKV + (value ? 2 * ((i + 1) % kStages) + 1 : 2 * (i % kStages)) * L::kTile;
    };
    const int n_here = it_hi - it_lo;

    if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;\n" ::);
    if (warp == 0) {
        // ---- producer: one lane per TMA box, so that the block-table reads of a tile are in flight together ----
        const int box_shift = 31 - __clz(p.box_rows), page_shift = 31 - __clz(p.page_size);
        const int per_tile_shift = (7 - box_shift) + (HD == 128 ? 1 : 0);          // boxes of a tile times 64-column halves
        const int which = lane >> per_tile_shift;    // 0: key, 1: value, above: idle lanes
        const int box = (lane & ((1 << per_tile_shift) - 1)) / (HD / 64), half = lane % (HD / 64);
        for (int i = 0; i < n_here + kLag; ++i) {
            const int st = i % kStages;
            const bool has = which == 0 ? i < n_here : (!SHARED && which == 1 && i >= 1);
            int row = 0;
            if (has) {
                const int it = it_lo + i - which;
                const bool pooled = it < n_pool;
                // A box that holds no entry any token of the block sees is never looked up (its page may have been given back): the
                // nearest box that does stands in for it.
                int key = first_key(it) + box * p.box_rows;
                if (pooled) key = min(key, nb_max - 1);
                else {
                    key = min(key, key_hi);                          // a request may be shorter than the kept first tokens
                    if (key >= keep) {
                        if (it < n_pool + n_kept) key = keep - 1;
                        else if (key + p.box_rows <= key_lo) key = key_lo;
                    }
                }
                key &= ~(p.box_rows - 1);
                const int slot = key >> page_shift;
                int page = slot < p.table_width ? table[slot] : -1;
                if (page < 0 || page >= p.num_pages) { atomicExch(p.err, 4); page = 0; }
                row = (((page * p.planes + (pooled ? 1 : 0)) * p.G + kvh) << page_shift) + (key & (p.page_size - 1));
            }
            if (lane == 0) {
                if (i >= kStages) mbar_wait(kv_empty + st, ((i / kStages) - 1) & 1, p.err);
                mbar_expect_tx(kv_full + st, L::kTile * (SHARED ? 1 : (i < n_here ? 1 : 0) + (i >= 1 ? 1 : 0)));
            }
            __syncwarp();
            if (has) {
                unsigned char* dst = which == 0 ? entry_tile(i, false) : entry_tile(i - 1, true);
                tma_load_2d(dst + half * 16384 + box * p.box_rows * 128, &map, kv_full + st, which * HD + half * 64, row);
            }
        }
    } else if (warp == 1) {
        // ---- tensor-core issue: the whole warp walks the list with values that are the same in all lanes, one lane issues ----
        constexpr uint32_t idesc_s = idesc_bf16(kEM, kEN, false);
        constexpr uint32_t idesc_pv = idesc_bf16(kEM, HD, true);
        constexpr uint32_t kTileStep = L::kTile >> 4;                         // in units of a descriptor's address
        const uint64_t q_desc = desc_sw128(smem_u32(sQ), 16, 1024), v_desc = desc_sw128(smem_u32(sKV), 16384, 1024);
        const uint32_t q_lo = static_cast<uint32_t>(q_desc), k_lo = static_cast<uint32_t>(desc_sw128(smem_u32(sKV), 16, 1024));
        const uint32_t v_lo = static_cast<uint32_t>(v_desc), k_hi = static_cast<uint32_t>(q_desc >> 32), v_hi = static_cast<uint32_t>(v_desc >> 32);
        const uint32_t t0 = same_in_warp(tmem);
        const int n = same_in_warp(n_here), end[2] = {same_in_warp(last_it[0] - it_lo), same_in_warp(last_it[1] - it_lo)};
        auto sees = [&](int x, int i) { return __any_sync(0xffffffffu, active(x, it_lo + i)) != 0; };
        auto issue_s = [&](int x, int i) {           // S(X) of list entry it_lo + i; its stage has been waited for
            const uint32_t ql = q_lo + x * kTileStep, kl = k_lo + (SHARED ? i % kStages : 2 * (i % kStages)) * kTileStep;
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < HD / 16; ++k) {
                    const uint32_t off = (k >> 2) * (16384 >> 4) + (k & 3) * 2;
                    umma(t0 + x * 128, desc_words(ql + off, k_hi), desc_words(kl + off, k_hi), idesc_s, k > 0 ? 1u : 0u);
                }
                tc_commit(s_ready + x);
            }
            __syncwarp();
        };
        int done[2] = {0, 0};                        // list entries of either query tile behind us
        bool now[2] = {sees(0, 0), sees(1, 0)};
        mbar_wait(kv_full + 0, 0, p.err);
#pragma unroll
        for (int x = 0; x < 2; ++x)
            if (now[x]) issue_s(x, 0);
        if (!SHARED && elect_one()) tc_commit(kv_empty + 0);
        __syncwarp();
        for (int i = 0; i < n; ++i) {
            const int next = i + 1, st = next % kStages;        // apart: load i + 1 brings these values and the next keys
            const bool soon[2] = {next < n && sees(0, next), next < n && sees(1, next)};
            if (!SHARED || next < n) mbar_wait(kv_full + st, (next / kStages) & 1, p.err);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                if (now[x]) {
                    const uint32_t vl = v_lo + (SHARED ? i % kStages : 2 * st + 1) * kTileStep, more = done[x] > 0 ? 1u : 0u;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {             // a half's product runs while the exponentials of the other are made
                        mbar_wait(p_ready + 2 * x + h, done[x] & 1, p.err);
                        tc_after();
                        if (elect_one()) {
#pragma unroll
                            for (int k = h * (kEN / 32); k < (h + 1) * (kEN / 32); ++k)   // P: 16 entries = 8 columns of packed pairs; V: 16 entries further down
                                umma_ts(t0 + 256 + x * HD, t0 + x * 128 + k * 8, desc_words(vl + k * (16 * 128 >> 4), v_hi), idesc_pv, k > 0 ? 1u : more);
                            if (h == 1 && i == end[x]) tc_commit(o_done + x);
                        }
                        __syncwarp();
                    }
                    ++done[x];
                }
                if (soon[x]) issue_s(x, next);
                now[x] = soon[x];
            }
            if (elect_one()) tc_commit(kv_empty + (SHARED ? i % kStages : st));
            __syncwarp();
        }
    }
    } else {                                         // ---- softmax: one thread per query row ----
        asm volatile("setmaxnreg.inc.sync.aligned.u32 224;\n" ::);
        const int x = (warp - 4) >> 2;               // query tile
        const int my_last = x ? last_it[1] : last_it[0], my_tok = x ? n_tok[1] : n_tok[0];
        const uint32_t my_s = x ? tS[1] : tS[0], my_o = x ? tO[1] : tO[0];
        const int quarter = warp & 3;                // the 32 lanes of tensor memory this warp may touch
        const int r = quarter * 32 + lane;           // row within the tile
        const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
        const bool has_keys = my_last >= 0;
        const int r_tok = row_tok(r), r_head = min(r - r_tok * g, g - 1);
        const int tok = x * tok_per_tile + min(r_tok, max(my_tok - 1, 0));
        const int row_pos = pos0 + tok;
        const int head = kvh * g + r_head;
        float m_ref = -INFINITY, l = 0.f;
        if (p.sink != nullptr && n_pieces == 1) { m_ref = p.sink[head] * kELog2e; l = 1.f; }
        const float scale_log2 = p.scale * kELog2e;
        if (has_keys) {
            const int row_lo = entry_first_visible(row_pos, p), row_nb = entry_visible_blocks(row_pos, p);
            const float* t_row = sT + r_head * p.table_stride + tok_per_tile + kEN;         // distance 0
            int done = 0;
            for (int it = it_lo; it <= my_last; ++it) {
                if (!active(x, it)) continue;
                const bool pooled = it < n_pool;
                const int key0 = first_key(it);
                mbar_wait(s_ready + x, done & 1, p.err);
                tc_after();
                uint32_t v[128];
#pragma unroll
                for (int c = 0; c < 4; ++c) tm_load32(my_s + lane_base + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&v[c * 32]));
                tm_wait_ld();
                const int hi = pooled ? row_nb - 1 : row_pos;
                auto mask = [&](uint32_t with) {
                    if (key0 + 127 > hi) {                                     // entries after the row's own
                        const int n_see = hi - key0 + 1;
#pragma unroll
                        for (int c = 0; c < 128; ++c) v[c] = c < n_see ? v[c] : with;
                    }
                    if (!pooled && key0 < row_lo) {                            // entries before the row's window, but for the kept ones
                        const int n_drop = row_lo - key0, n_keep = keep - key0;
#pragma unroll
                        for (int c = 0; c < 128; ++c) v[c] = (c < n_drop && c >= n_keep) ? with : v[c];
                    }
                };
                if (TERMS) {
                    if (p.softcap > 0.f) {
                        mask(0u);               // what a former holder left in a page must not choose between the two forms below
                        const float k = p.scale / p.softcap, back = p.softcap * kELog2e;
                        float top = 0.f;
#pragma unroll
                        for (int c = 0; c < 128; ++c) top = fmaxf(top, fabsf(__uint_as_float(v[c])));
                        if (__any_sync(0xffffffffu, top * fabsf(k) > 0.4f)) {
#pragma unroll
                            for (int c = 0; c < 128; ++c) v[c] = __float_as_uint(tanh_exponential(__uint_as_float(v[c]) * k) * back);
                        } else {
                            const float2 k2 = make_float2(k, k), back2 = make_float2(back, back);
#pragma unroll
                            for (int c = 0; c < 128; c += 2) {
                                const float2 s = __fmul2_rn(tanh_small2(__fmul2_rn(make_float2(__uint_as_float(v[c]), __uint_as_float(v[c + 1])), k2)), back2);
                                v[c] = __float_as_uint(s.x);
                                v[c + 1] = __float_as_uint(s.y);
                            }
                        }
                    } else {
                        const float2 k2 = make_float2(scale_log2, scale_log2);
#pragma unroll
                        for (int c = 0; c < 128; c += 2) {
                            const float2 s = __fmul2_rn(make_float2(__uint_as_float(v[c]), __uint_as_float(v[c + 1])), k2);
                            v[c] = __float_as_uint(s.x);
                            v[c + 1] = __float_as_uint(s.y);
                        }
                    }
                    if (p.table_len > 0 && !pooled) {
                        const int d0 = row_pos - key0;                          // distance of the tile's first key
                        if (__all_sync(0xffffffffu, d0 - (kEN - 1) >= p.table_len - 1)) {
                            const float far = t_row[p.table_len - 1];
#pragma unroll
                            for (int c = 0; c < 128; ++c) v[c] = __float_as_uint(__uint_as_float(v[c]) + far);
                        } else {
                            const float* at = t_row + d0;
#pragma unroll
                            for (int c = 0; c < 128; ++c) v[c] = __float_as_uint(__uint_as_float(v[c]) + at[-c]);
                        }
                    }
                }
                mask(0xff800000u);                                             // -inf
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};       // four chains of three-input maxima
#pragma unroll
                for (int c = 0; c < 128; c += 8) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) mx[k] = max3(mx[k], __uint_as_float(v[c + 2 * k]), __uint_as_float(v[c + 2 * k + 1]));
                }
                float m_tile = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                if (!TERMS) m_tile *= scale_log2;
                const float m_new = fmaxf(m_ref, m_tile);
                if (__any_sync(0xffffffffu, m_new > m_ref)) {
                    const float m_use = m_new == -INFINITY ? 0.f : m_new;
                    const float factor = ex2(m_ref - m_use);             // 2^(-inf) = 0 before the first key
                    m_ref = m_new;
                    l *= factor;
                    if (done > 0) {                                       // O(X) holds the products up to here, all done
#pragma unroll
                        for (int c = 0; c < HD; c += 32) {
                            uint32_t o[32];
                            tm_load32(my_o + lane_base + c, o);
                            tm_wait_ld();
#pragma unroll
                            for (int k = 0; k < 32; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * factor);
                            tm_store32(my_o + lane_base + c, o);
                        }
                    }
                }
                // Entries that no token of the block sees have probability 0, but what the page holds there (a former holder's
                // Inf, a NaN) times 0 would be NaN: thread r clears row r of the tile the product P V reads.  (The threads of the
                // other query tile may do the same; they write the same zeros.)
                const bool dirty = pooled ? key0 + kEN > nb_max : (key0 + kEN - 1 > key_hi || (key0 < key_lo && keep < key0 + kEN));
                if (dirty) {
                    const int i = it - it_lo, load = i + kLag;
                    mbar_wait(kv_full + load % kStages, (load / kStages) & 1, p.err);
                    const int j = key0 + r;
                    if (pooled ? j >= nb_max : (j > key_hi || (j < key_lo && j >= keep))) {
                        __nv_bfloat16* rows = reinterpret_cast<__nv_bfloat16*>(entry_tile(i, true));
#pragma unroll
                        for (int c = 0; c < CPR; ++c) *reinterpret_cast<uint4*>(rows + entry_off(r, c)) = make_uint4(0u, 0u, 0u, 0u);
                    }
                    fence_async_smem();                                       // the tensor core reads through the async proxy
                }
                const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
                const float2 scale2 = make_float2(scale_log2, scale_log2), neg_m2 = make_float2(-m_use, -m_use);
                float2 sum2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t packed[32];
#pragma unroll
                    for (int k = 0; k < 32; ++k) {
                        const int c = h * 64 + 2 * k;
                        const float2 s = make_float2(__uint_as_float(v[c]), __uint_as_float(v[c + 1]));
                        const float2 arg = TERMS ? __fadd2_rn(s, neg_m2) : __ffma2_rn(s, scale2, neg_m2);
                        const float2 pr = make_float2(ex2(arg.x), ex2(arg.y));
                        sum2[k & 1] = __fadd2_rn(sum2[k & 1], pr);
                        __nv_bfloat162 hh = __floats2bfloat162_rn(pr.x, pr.y);
                        packed[k] = *reinterpret_cast<uint32_t*>(&hh);
                    }
                    tm_store32(my_s + lane_base + h * 32, packed);     // P over the first 64 columns of S
                    tm_wait_st();
                    tc_before();
                    mbar_arrive(p_ready + 2 * x + h);
                }
                l += (sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y);
                ++done;
            }
        }
        // the gate's row is asked for while the last product runs
        const bool store = has_keys && n_pieces == 1;
        uint4 gate_row[DV / 8];
        float inv = l > 0.f ? p.out_scale / l : 0.f;
        if (store && p.gate != nullptr) {
            const __nv_bfloat16* grow = p.gate + static_cast<int64_t>(cu0 + q0 + tok) * p.gate_stride;
            if (p.gate_element) {
#pragma unroll
                for (int c = 0; c < DV / 8; ++c) gate_row[c] = *reinterpret_cast<const uint4*>(grow + head * DV + c * 8);
            } else {
                inv *= 1.f / (1.f + __expf(-__bfloat162float(grow[head])));
            }
        }
        if (has_keys) {
            mbar_wait(o_done + x, 0, p.err);
            tc_after();
        }
        // The rows go through shared memory (over the query tile, which no product reads any more, in its swizzled layout) so that the
        // stores to global memory are whole rows side by side.
        __nv_bfloat16* stage = reinterpret_cast<__nv_bfloat16*>(sQ + x * L::kTile);
        if (store) {
#pragma unroll
            for (int c0 = 0; c0 < DV; c0 += 32) {
                uint32_t o[32];
                tm_load32(my_o + lane_base + c0, o);
                tm_wait_ld();
                if (p.gate != nullptr && p.gate_element) {
#pragma unroll
                    for (int k = 0; k < 32; k += 8) {
                        const __nv_bfloat162* z2 = reinterpret_cast<const __nv_bfloat162*>(&gate_row[(c0 + k) / 8]);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float2 z = __bfloat1622float2(z2[e]);
                            o[k + 2 * e] = __float_as_uint(__uint_as_float(o[k + 2 * e]) * __fdividef(1.f, 1.f + __expf(-z.x)));
                            o[k + 2 * e + 1] = __float_as_uint(__uint_as_float(o[k + 2 * e + 1]) * __fdividef(1.f, 1.f + __expf(-z.y)));
                        }
                    }
                }
#pragma unroll
                for (int k = 0; k < 32; k += 8) {
                    uint4 t;
                    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&t);
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        h[e] = __floats2bfloat162_rn(__uint_as_float(o[k + 2 * e]) * inv, __uint_as_float(o[k + 2 * e + 1]) * inv);
                    *reinterpret_cast<uint4*>(stage + entry_off(r, (c0 + k) >> 3)) = t;
                }
            }
        } else if (n_pieces > 1) {
            // ---- one of several pieces: leave its share for the merge; rows lie side by side, a warp writes whole lines ----
            float* mine = p.part_o + (static_cast<int64_t>(part_slot) * 2 + x) * (DV * 128) + r;
            float* mine_ml = p.part_ml + (static_cast<int64_t>(part_slot) * 2 + x) * 256 + r;
            if (has_keys) {
#pragma unroll
                for (int c0 = 0; c0 < DV; c0 += 32) {
                    uint32_t o[32];
                    tm_load32(my_o + lane_base + c0, o);
                    tm_wait_ld();
#pragma unroll
                    for (int c = 0; c < 32; ++c) __stcg(mine + (c0 + c) * 128, __uint_as_float(o[c]));
                }
            }
            __stcg(mine_ml, has_keys ? m_ref : -INFINITY);
            __stcg(mine_ml + 128, has_keys ? l : 0.f);          // no sum: the piece had no key for this row
        }
        if (store) {
            asm volatile("bar.sync %0, 128;\n" ::"r"(2 + x) : "memory");       // the 128 threads of this query tile
            __nv_bfloat16* out_base = p.out + (static_cast<int64_t>(cu0 + q0) + x * tok_per_tile) * p.out_stride + kvh * g * DV;
            constexpr int OCR = DV / 8;                                        // 16-byte chunks of an output row
#pragma unroll 4
            for (int i = r; i < kEM * OCR; i += 128) {
                const int row = i / OCR, c = i % OCR;
                const int t = row_tok(row), h = row - t * g;
                if (t < my_tok)
                    *reinterpret_cast<uint4*>(out_base + static_cast<int64_t>(t) * p.out_stride + h * DV + c * 8) =
                        *reinterpret_cast<const uint4*>(stage + entry_off(row, c));
            }
        }
    }
    tc_before();
    __syncthreads();
    if (warp == 1) {
        tc_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
    }
}

// Adds up the shares of query blocks that attn_entries_tcgen05_kernel cut into pieces and stores their rows.  Grid: (query block * kv
// head, query tile, 32 columns of the head); thread r owns row r of the query tile.  Piece k weighs 2^(its reference maximum - the
// largest of them); shares are added in the order of the pieces, the sink joins last.
__global__ void __launch_bounds__(128)
attn_entries_merge_kernel(const EntryAttnParams p, const int dv) {
    constexpr int kRowBytes = 64 + 16;                              // 32 bf16 of a row, padded against bank conflicts
    __shared__ __align__(16) unsigned char stage[128 * kRowBytes];
    pdl_trigger();
    const int g = p.H / p.G;
    const int tok_per_tile = kEM / g, tok_per_block = 2 * tok_per_tile;
    const int block_id = blockIdx.x / p.G, kvh = blockIdx.x - block_id * p.G;
    const int x = blockIdx.y, c0 = blockIdx.z * 32, r = threadIdx.x, lane = threadIdx.x & 31;
    int q0 = 0, q_len = 0, cu0 = 0;
    const int seq = entry_find_block(p, block_id, tok_per_block, lane, q0, q_len, cu0);
    if (seq < 0) return;
    const int n_tok = max(0, min(tok_per_tile, q_len - q0 - x * tok_per_tile));
    if (n_tok == 0) return;
    pdl_wait();
    const int n_pieces = min(p.piece_counts[blockIdx.x], kEMaxPieces);
    if (n_pieces <= 1) return;                                      // the block stored its rows itself
    const int64_t first = static_cast<int64_t>(blockIdx.x) * p.pieces;
    float w[kEMaxPieces], sum[kEMaxPieces];
#pragma unroll
    for (int k = 0; k < kEMaxPieces; ++k) {
        const float* ml = p.part_ml + ((first + k) * 2 + x) * 256 + r;
        w[k] = k < n_pieces ? __ldcg(ml) : -INFINITY;
        sum[k] = k < n_pieces ? __ldcg(ml + 128) : 0.f;
    }
    const int t_r = min(r / g, n_tok - 1), head = kvh * g + min(r - r / g * g, g - 1);
    const int64_t t_abs = static_cast<int64_t>(cu0 + q0) + x * tok_per_tile + t_r;
    float m_all = p.sink != nullptr ? p.sink[head] * kELog2e : -INFINITY, l = 0.f;
#pragma unroll
    for (int k = 0; k < kEMaxPieces; ++k) {
        if (sum[k] == 0.f) w[k] = -INFINITY;                        // a piece without a key for this row; a NaN stays
        m_all = fmaxf(m_all, w[k]);
    }
#pragma unroll
    for (int k = 0; k < kEMaxPieces; ++k) {
        w[k] = sum[k] == 0.f ? 0.f : ex2(w[k] - m_all);
        l = __fadd_rn(l, __fmul_rn(sum[k], w[k]));
    }
    if (p.sink != nullptr) l += ex2(p.sink[head] * kELog2e - m_all);
    float acc[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) acc[c] = 0.f;
#pragma unroll
    for (int k = 0; k < kEMaxPieces; ++k) {
        if (sum[k] == 0.f) continue;                                // never written
        const float* share = p.part_o + ((first + k) * 2 + x) * (static_cast<int64_t>(dv) * 128) + static_cast<int64_t>(c0) * 128 + r;
#pragma unroll
        for (int c = 0; c < 32; ++c) acc[c] = __fadd_rn(acc[c], __fmul_rn(__ldcg(share + c * 128), w[k]));
    }
    float inv = l == 0.f ? 0.f : p.out_scale / l;
    if (p.gate != nullptr) {
        const __nv_bfloat16* grow = p.gate + t_abs * p.gate_stride;
        if (p.gate_element) {
#pragma unroll
            for (int c = 0; c < 32; ++c) acc[c] *= __fdividef(1.f, 1.f + __expf(-__bfloat162float(grow[head * dv + c0 + c])));
        } else {
            inv *= 1.f / (1.f + __expf(-__bfloat162float(grow[head])));
        }
    }
#pragma unroll
    for (int k = 0; k < 32; k += 8) {
        uint4 t;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&t);
#pragma unroll
        for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(acc[k + 2 * e] * inv, acc[k + 2 * e + 1] * inv);
        *reinterpret_cast<uint4*>(stage + r * kRowBytes + k * 2) = t;
    }
    __syncthreads();
    // four threads store the 64 bytes of a row
    __nv_bfloat16* out_base = p.out + (static_cast<int64_t>(cu0 + q0) + x * tok_per_tile) * p.out_stride + kvh * g * dv + c0;
    const int chunk = r & 3;
#pragma unroll
    for (int pass = 0; pass < 4; ++pass) {
        const int row = pass * 32 + (r >> 2);
        const int t = row / g, h = row - t * g;
        if (t < n_tok)
            *reinterpret_cast<uint4*>(out_base + static_cast<int64_t>(t) * p.out_stride + h * dv + chunk * 8) =
                *reinterpret_cast<const uint4*>(stage + row * kRowBytes + chunk * 16);
    }
}

// ---- host side ------------------------------------------------------------------------------------------------

// Floats per head of the distance table (0: none): the distances, what stands for distances below 0 and the copies of the last one;
// rows of neighbouring heads start 32 / g banks apart.
static int entry_table_stride(int table_len, int g) {
    if (table_len <= 0) return 0;
    const int len = kEM / g + kEN + table_len + kEPadHigh;
    return (len + 31) / 32 * 32 + (g < 32 ? 32 / g : 1);
}

constexpr size_t kEMaxShared = 232448;        // 227 KB

template <int HD, int DV, bool SHARED, bool TERMS>
int launch_entries(const CUtensorMap& map, const EntryAttnParams& p, int num_tiles, cudaStream_t stream) {
    const size_t smem = EntrySmem<HD>::kBytes + static_cast<size_t>(p.H / p.G) * p.table_stride * sizeof(float);
    static bool set = false;
    if (!set) {
        if (cudaFuncSetAttribute(attn_entries_tcgen05_kernel<HD, DV, SHARED, TERMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEMaxShared) != cudaSuccess)
            return launch_status();
        set = true;
    }
    dim3 grid(static_cast<unsigned>(p.G), static_cast<unsigned>(num_tiles), static_cast<unsigned>(p.pieces));
    launch_kernel(attn_entries_tcgen05_kernel<HD, DV, SHARED, TERMS>, grid, dim3(kEThreads), smem, stream, map, p);
    const int launched = launch_status();
    if (launched != CVB_OK || p.pieces == 1) return launched;
    launch_kernel(attn_entries_merge_kernel, dim3(static_cast<unsigned>(num_tiles * p.G), 2, static_cast<unsigned>(DV / 32)), dim3(128), 0, stream, p, DV);
    return launch_status();
}

}  // namespace cvb

using namespace cvb;

// Whether the kernel takes the shape: key and value sizes, group, page size, and a distance table (`table_len` entries a head, 0: none)
// that fits beside the tiles.
extern "C" int cvb_attn_entries_supported(int H, int G, int dk, int dv, int shared, int page_size, int table_len) {
    if (H <= 0 || G <= 0 || H % G || H / G > 128) return 0;
    if (dk != 64 && dk != 128) return 0;
    if (shared ? !(dv == dk || (dk == 128 && dv == 96)) : dv != dk) return 0;
    if (shared && table_len > 0) return 0;
    if (page_size < 16 || (page_size & (page_size - 1)) != 0 || table_len < 0 || table_len > (1 << 20)) return 0;
    const size_t tiles = dk == 128 ? EntrySmem<128>::kBytes : EntrySmem<64>::kBytes;
    return tiles + static_cast<size_t>(H / G) * entry_table_stride(table_len, H / G) * sizeof(float) <= kEMaxShared ? 1 : 0;
}

// Floats of scratch that `pieces` > 1 needs for num_tiles query blocks: outputs, maxima and sums of every piece.
extern "C" int64_t cvb_attn_entries_scratch_floats(int num_tiles, int G, int dv, int pieces) {
    return static_cast<int64_t>(num_tiles) * G * pieces * 2 * (dv + 2) * 128;
}

// What a layer asks of the kernel whatever the step.
struct EntryAttnShape {
    int H, G, dk, dv, shared, page_size, planes, chunk, window, pool, keep, table_len;
    float scale, softcap, out_scale;
};

// num_tiles: per request ceil(tokens / (2 * (128 / group))) query blocks.  `table_len` > 0: distances 0 .. table_len - 1 have an entry,
// of `bias` [H, bias_len] (bias_len = table_len) or of r1, r2; larger distances take the last one (with r1, r2 the mask must rule them
// out).  With pieces > 1 a query block of at least 2 * min_rounds tiles is worked on by up to `pieces` blocks.
extern "C" int cvb_attn_entries_tcgen05(const EntryAttnShape* shape, void* out, int out_stride, const void* q, int q_stride, const void* pages,
                                        int num_pages, const int* block_tables, int table_width, const int* cu_seqlens, const int* positions, int S,
                                        int num_tiles, const float* bias, const float* r1, const float* r2, const float* sink, const void* gate,
                                        int bias_len, int gate_stride, int gate_element, int pieces, int min_rounds, float* scratch,
                                        int64_t scratch_floats, int* piece_counts, int* err_flag, cudaStream_t stream) {
    const auto [H, G, dk, dv, shared, page_size, planes, chunk, window, pool, keep, table_len, scale, softcap, out_scale] = *shape;
    if (num_tiles == 0) return CVB_OK;
    if (num_tiles < 0 || num_tiles > 65535 || S <= 0 || table_width <= 0 || num_pages <= 0 || planes < 1 || planes > 2 || bias_len < 0) return CVB_E_SIZE;
    if (chunk < 0 || window < 0 || pool < 0 || keep < 0 || (pool > 0 && planes != 2)) return CVB_E_SIZE;
    if ((pool > 0 || keep > 0) && window == 0) return CVB_E_SHAPE;  // they stand beside a window
    if (!cvb_attn_entries_supported(H, G, dk, dv, shared, page_size, table_len)) return CVB_E_UNSUPPORTED;
    if ((bias != nullptr && bias_len != table_len) || ((bias != nullptr || r1 != nullptr) != (table_len > 0)) || (r1 != nullptr) != (r2 != nullptr)) return CVB_E_SHAPE;
    const bool terms = softcap > 0.f || table_len > 0;
    if (shared && terms) return CVB_E_UNSUPPORTED;
    if (!terms && !(scale > 0.f)) return CVB_E_UNSUPPORTED;         // such scores are masked and their maximum taken before the scale
    if (q_stride < H * dk || out_stride < H * dv || q_stride % 8 || out_stride % 8) return CVB_E_ALIGN;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(pages) | reinterpret_cast<uintptr_t>(out)) & 15) return CVB_E_ALIGN;
    if (gate != nullptr && gate_element && (gate_stride % 8 || (reinterpret_cast<uintptr_t>(gate) & 15))) return CVB_E_ALIGN;
    if (static_cast<int64_t>(num_pages) * planes * G * page_size > 2147483647LL) return CVB_E_SIZE;
    if (pieces < 1 || pieces > kEMaxPieces || min_rounds < 1) return CVB_E_SIZE;
    if (static_cast<int64_t>(num_tiles) * G * pieces > 2147483647LL) return CVB_E_SIZE;
    if (pieces > 1 && (!scratch || !piece_counts || scratch_floats < cvb_attn_entries_scratch_floats(num_tiles, G, dv, pieces))) return CVB_E_SCRATCH;
    EntryAttnParams p{};
    p.out = (__nv_bfloat16*)out; p.q = (const __nv_bfloat16*)q; p.gate = (const __nv_bfloat16*)gate;
    p.bias = bias; p.r1 = r1; p.r2 = r2; p.sink = sink;
    p.block_tables = block_tables; p.cu_seqlens = cu_seqlens; p.positions = positions;
    p.q_stride = q_stride; p.out_stride = out_stride; p.gate_stride = gate_stride; p.gate_element = gate_element;
    p.table_width = table_width; p.S = S; p.H = H; p.G = G; p.page_size = page_size; p.planes = planes; p.num_pages = num_pages;
    p.box_rows = page_size < 64 ? page_size : 64;
    p.chunk = chunk; p.window = window; p.pool = pool; p.keep = keep;
    p.table_len = table_len; p.table_stride = entry_table_stride(table_len, H / G); p.bias_len = bias_len;
    p.scale = scale; p.softcap = softcap; p.out_scale = out_scale; p.err = err_flag;
    p.pieces = pieces; p.min_rounds = min_rounds; p.piece_counts = piece_counts; p.part_o = scratch;
    p.part_ml = scratch ? scratch + static_cast<int64_t>(num_tiles) * G * pieces * 2 * dv * 128 : nullptr;
    CUtensorMap map;
    const int rc = cached_bf16_map(&map, pages, static_cast<int64_t>(num_pages) * planes * G * page_size, shared ? dk : dk + dv, 64, p.box_rows);
    if (rc != CVB_OK) return rc;
    if (shared) {
        if (dk == 64) return launch_entries<64, 64, true, false>(map, p, num_tiles, stream);
        return dv == 96 ? launch_entries<128, 96, true, false>(map, p, num_tiles, stream) : launch_entries<128, 128, true, false>(map, p, num_tiles, stream);
    }
    if (dk == 64) return terms ? launch_entries<64, 64, false, true>(map, p, num_tiles, stream) : launch_entries<64, 64, false, false>(map, p, num_tiles, stream);
    return terms ? launch_entries<128, 128, false, true>(map, p, num_tiles, stream) : launch_entries<128, 128, false, false>(map, p, num_tiles, stream);
}
