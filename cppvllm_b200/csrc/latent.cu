// What stands around attention over a cache of latent vectors (one vector per token, shared by all heads):
//
//   latent_prep      : per token, from the packed output of the down projections:
//                        cq = T( a / sqrt(mean(a^2) + eps) * wq )                 the query latent, normed
//                        c  = T( b / sqrt(mean(b^2) + eps) * wk )                 the key/value latent, normed
//                        kr = T( rot_p(r) )                                       the positional key part, turned by the token's position
//                      and [c | kr] written into the token's slot of the cache pages [page, slot in page, rank + rot].
//                      Either half may be left out (a layer that reads another layer's cache writes none).
//   latent_q_assemble: the query that the attention kernel reads, per token and head: [q_abs | rot_p(q_rot)], where q_abs
//                      (the unrotated query taken through the key up-projection, laid out [head, token, rank]) comes from a
//                      batched product and q_rot is the head's positional part inside the packed query projection.
//   latent_q_turn    : the same where the batched product has written q_abs to its place already: the turned parts alone.
//   head_gate        : att[t, h, :] = T( o[h, t, :] * sigmoid(g[t, h]) ): one gate per token and head, and the move from the
//                      batched product's [head, token, :] to rows of concatenated heads.  With `per_element` the gate has
//                      one number per element of the concatenated heads: att[t, i] = T( o[..] * sigmoid(g[t, i]) ).
//
// The rotation pairs element 2i with element 2i+1 of the first `rot` elements (cos and sin tables [positions, rot / 2],
// float); elements behind them pass unchanged.  Norm statistics and the rotation are float.
#include "common.cuh"

namespace cvb {

constexpr int kLatentThreads = 128;

template <typename T>
__device__ __forceinline__ void norm_part(T* __restrict__ out, const T* __restrict__ in, const float* __restrict__ w, int n,
                                          float eps, float* scratch) {
    float ss = 0.f;
    for (int i = threadIdx.x; i < n; i += kLatentThreads) {
        const float v = to_float(in[i]);
        ss = fmaf(v, v, ss);
    }
    ss = block_sum(ss, scratch);
    const float inv = 1.f / sqrtf(ss / static_cast<float>(n) + eps);
    for (int i = threadIdx.x; i < n; i += kLatentThreads) out[i] = from_float<T>(to_float(in[i]) * inv * w[i]);
}

// out[0 .. width): in[0 .. width) with the first `rot` elements turned by the angle tables' row.
template <typename T>
__device__ __forceinline__ void rotate_part(T* __restrict__ out, const T* __restrict__ in, const float* __restrict__ cs,
                                            const float* __restrict__ sn, int rot, int width) {
    for (int i = threadIdx.x; i < width; i += kLatentThreads) {
        float v = to_float(in[i]);
        if (i < rot) {
            const float c = cs[i >> 1], s = sn[i >> 1];
            const float other = to_float(in[i ^ 1]);
            v = (i & 1) ? v * c + other * s : v * c - other * s;
        }
        out[i] = from_float<T>(v);
    }
}

template <typename T>
__global__ void __launch_bounds__(kLatentThreads)
latent_prep_kernel(T* __restrict__ cq_out, T* __restrict__ pages, const T* __restrict__ packed, int stride, int q_off, int q_rank,
                   const float* __restrict__ wq, int kv_off, int rank, int rot_width, int rot, const float* __restrict__ wk,
                   const float* __restrict__ cos_t, const float* __restrict__ sin_t, int max_pos, const int* __restrict__ positions,
                   const int* __restrict__ slots, int64_t total_slots, float eps, int* __restrict__ err) {
    pdl_trigger();
    pdl_wait();
    __shared__ float scratch[32];
    const int64_t t = blockIdx.x;
    const T* row = packed + t * stride;
    if (cq_out != nullptr) norm_part(cq_out + t * q_rank, row + q_off, wq, q_rank, eps, scratch);
    if (pages == nullptr) return;
    const int slot = slots[t];
    if (slot < 0) return;
    if (slot >= total_slots) {
        if (threadIdx.x == 0) atomicExch(err, 2);
        return;
    }
    int p = positions[t];
    if (p < 0 || p >= max_pos) {
        if (threadIdx.x == 0) atomicExch(err, 3);
        p = p < 0 ? 0 : max_pos - 1;
    }
    T* entry = pages + static_cast<int64_t>(slot) * (rank + rot_width);
    norm_part(entry, row + kv_off, wk, rank, eps, scratch);
    rotate_part(entry + rank, row + kv_off + rank, cos_t + static_cast<int64_t>(p) * (rot / 2), sin_t + static_cast<int64_t>(p) * (rot / 2),
                rot, rot_width);
}

template <typename T>
__global__ void __launch_bounds__(kLatentThreads)
latent_q_assemble_kernel(T* __restrict__ q_out, const T* __restrict__ q_abs, const T* __restrict__ q, int q_stride, int H, int nope,
                         int rank, int rot_width, int rot, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                         int max_pos, const int* __restrict__ positions, int T_total, int* __restrict__ err) {
    pdl_trigger();
    pdl_wait();
    const int64_t t = blockIdx.x;
    const int h = blockIdx.y;
    int p = positions[t];
    if (p < 0 || p >= max_pos) {
        if (threadIdx.x == 0) atomicExch(err, 3);
        p = p < 0 ? 0 : max_pos - 1;
    }
    T* dst = q_out + (t * H + h) * (rank + rot_width);
    const T* src = q_abs + (static_cast<int64_t>(h) * T_total + t) * rank;
    for (int i = threadIdx.x; i < rank; i += kLatentThreads) dst[i] = src[i];
    rotate_part(dst + rank, q + t * q_stride + h * (nope + rot_width) + nope, cos_t + static_cast<int64_t>(p) * (rot / 2),
                sin_t + static_cast<int64_t>(p) * (rot / 2), rot, rot_width);
}

template <typename T>
__global__ void __launch_bounds__(kLatentThreads)
latent_q_turn_kernel(T* __restrict__ q_out, const T* __restrict__ q, int q_stride, int H, int nope, int rank, int rot_width, int rot,
                     const float* __restrict__ cos_t, const float* __restrict__ sin_t, int max_pos, const int* __restrict__ positions,
                     int* __restrict__ err) {
    pdl_trigger();
    pdl_wait();
    const int64_t t = blockIdx.x;
    int p = positions[t];
    if (p < 0 || p >= max_pos) {
        if (threadIdx.x == 0) atomicExch(err, 3);
        p = p < 0 ? 0 : max_pos - 1;
    }
    const float* cs = cos_t + static_cast<int64_t>(p) * (rot / 2);
    const float* sn = sin_t + static_cast<int64_t>(p) * (rot / 2);
    for (int i = blockIdx.y * kLatentThreads + threadIdx.x; i < H * rot_width; i += gridDim.y * kLatentThreads) {
        const int h = i / rot_width, e = i - h * rot_width;
        const T* in = q + t * q_stride + h * (nope + rot_width) + nope;
        float v = to_float(in[e]);
        if (e < rot) {
            const float c = cs[e >> 1], s = sn[e >> 1], other = to_float(in[e ^ 1]);
            v = (e & 1) ? v * c + other * s : v * c - other * s;
        }
        q_out[(t * H + h) * (rank + rot_width) + rank + e] = from_float<T>(v);
    }
}

// The same by 16 bytes per thread, where the turned part, what lies in front of it and the rotation are whole pieces
// (2,048 tokens of 16 heads, 32 elements each: 9.7 -> 3.0 us).
template <typename T>
__global__ void __launch_bounds__(256)
latent_q_turn_vec_kernel(T* __restrict__ q_out, const T* __restrict__ q, int q_stride, int H, int nope, int rank, int rot_width, int rot,
                         const float* __restrict__ cos_t, const float* __restrict__ sin_t, int max_pos, const int* __restrict__ positions,
                         int total, int* __restrict__ err) {
    pdl_trigger();
    pdl_wait();
    constexpr int N = 16 / sizeof(T);
    const int chunks = rot_width / N, per = H * chunks;
    for (int i = blockIdx.x * 256 + threadIdx.x; i < total; i += gridDim.x * 256) {
        const int t = i / per, r = i - t * per, h = r / chunks, e = (r - h * chunks) * N;
        alignas(16) T v[N];
        *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(q + static_cast<int64_t>(t) * q_stride + h * (nope + rot_width) + nope + e);
        if (e < rot) {
            int p = positions[t];
            if (p < 0 || p >= max_pos) {
                atomicExch(err, 3);
                p = p < 0 ? 0 : max_pos - 1;
            }
            const float* cs = cos_t + static_cast<int64_t>(p) * (rot / 2) + e / 2;
            const float* sn = sin_t + static_cast<int64_t>(p) * (rot / 2) + e / 2;
#pragma unroll
            for (int k = 0; k < N; k += 2) {
                const float x = to_float(v[k]), y = to_float(v[k + 1]), c = cs[k / 2], s = sn[k / 2];
                v[k] = from_float<T>(x * c - y * s);
                v[k + 1] = from_float<T>(y * c + x * s);
            }
        }
        *reinterpret_cast<uint4*>(q_out + (static_cast<int64_t>(t) * H + h) * (rank + rot_width) + rank + e) = *reinterpret_cast<const uint4*>(v);
    }
}

template <typename T>
__global__ void __launch_bounds__(kLatentThreads)
head_gate_kernel(T* __restrict__ out, int out_stride, const T* __restrict__ o, const T* __restrict__ gate, int gate_stride, int H, int vd, int T_total,
                 int per_element) {
    pdl_trigger();
    pdl_wait();
    const int64_t t = blockIdx.x;
    for (int i = blockIdx.y * kLatentThreads + threadIdx.x; i < H * vd; i += gridDim.y * kLatentThreads) {
        const int h = i / vd, j = i - h * vd;
        const float z = to_float(gate[t * gate_stride + (per_element ? i : h)]);
        out[t * out_stride + i] = from_float<T>(to_float(o[(static_cast<int64_t>(h) * T_total + t) * vd + j]) * (1.f / (1.f + expf(-z))));
    }
}

// The same by 16 bytes per thread and four of them in flight, where a head's values are whole pieces and every row starts on one: element by
// element with a block per 128 of them, 2,048 tokens of 16 heads of 128 took 35 us for 17 MB; now 7.3.
template <typename T>
__global__ void __launch_bounds__(256)
head_gate_vec_kernel(T* __restrict__ out, int out_stride, const T* __restrict__ o, const T* __restrict__ gate, int gate_stride, int H, int vd, int T_total,
                     int per_element, int total) {
    pdl_trigger();
    pdl_wait();
    constexpr int N = 16 / sizeof(T), K = 4;
    const int chunks = vd / N, per = H * chunks, step = gridDim.x * 256;
    for (int i0 = blockIdx.x * 256 + threadIdx.x; i0 < total; i0 += K * step) {
        alignas(16) T x[K][N], z[K][N];
        int64_t dst[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int i = i0 + k * step;
            if (i < total) {
                const int t = i / per, r = i - t * per, h = r / chunks, c = (r - h * chunks) * N;
                dst[k] = static_cast<int64_t>(t) * out_stride + h * vd + c;
                *reinterpret_cast<uint4*>(x[k]) = *reinterpret_cast<const uint4*>(o + (static_cast<int64_t>(h) * T_total + t) * vd + c);
                const T* g = gate + static_cast<int64_t>(t) * gate_stride;
                if (per_element) *reinterpret_cast<uint4*>(z[k]) = *reinterpret_cast<const uint4*>(g + h * vd + c);
                else z[k][0] = g[h];
            }
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (i0 + k * step < total) {
                float f = per_element ? 0.f : 1.f / (1.f + expf(-to_float(z[k][0])));
#pragma unroll
                for (int e = 0; e < N; ++e) {
                    if (per_element) f = 1.f / (1.f + expf(-to_float(z[k][e])));
                    x[k][e] = from_float<T>(to_float(x[k][e]) * f);
                }
                *reinterpret_cast<uint4*>(out + dst[k]) = *reinterpret_cast<const uint4*>(x[k]);
            }
        }
    }
}

}  // namespace cvb

using namespace cvb;

extern "C" int cvb_latent_prep(void* cq_out, void* pages, const void* packed, int T, int stride, int q_off, int q_rank, const float* wq,
                               int kv_off, int rank, int rot_width, int rot, const float* wk, const float* cos_t, const float* sin_t,
                               int max_pos, const int* positions, const int* slots, int64_t total_slots, float eps, int dtype,
                               int* err_flag, cudaStream_t stream) {
    if (T == 0) return CVB_OK;
    if (T < 0 || stride <= 0) return CVB_E_SIZE;
    if (cq_out != nullptr && (q_rank <= 0 || q_off < 0 || q_off + q_rank > stride || wq == nullptr)) return CVB_E_SHAPE;
    if (pages != nullptr && (rank <= 0 || rot_width < 0 || rot < 0 || rot > rot_width || rot % 2 || kv_off < 0 ||
                             kv_off + rank + rot_width > stride || wk == nullptr || (rot > 0 && (cos_t == nullptr || sin_t == nullptr)) ||
                             max_pos <= 0 || total_slots <= 0))
        return CVB_E_SHAPE;
#define CALL(TY) launch_kernel(latent_prep_kernel<TY>, dim3(T), dim3(kLatentThreads), 0, stream, (TY*)cq_out, (TY*)pages, \
                               (const TY*)packed, stride, q_off, q_rank, wq, kv_off, rank, rot_width, rot, wk, cos_t, sin_t, max_pos, \
                               positions, slots, total_slots, eps, err_flag)
    CVB_DISPATCH_DTYPE(dtype, CALL);
#undef CALL
    return launch_status();
}

extern "C" int cvb_latent_q_assemble(void* q_out, const void* q_abs, const void* q, int T, int q_stride, int H, int nope, int rank,
                                     int rot_width, int rot, const float* cos_t, const float* sin_t, int max_pos, const int* positions,
                                     int dtype, int* err_flag, cudaStream_t stream) {
    if (T == 0) return CVB_OK;
    if (T < 0 || H <= 0 || H > 65535 || nope <= 0 || rank <= 0 || rot_width < 0 || max_pos <= 0) return CVB_E_SIZE;
    if (rot < 0 || rot > rot_width || rot % 2 || q_stride < H * (nope + rot_width)) return CVB_E_SHAPE;
#define CALL(TY) launch_kernel(latent_q_assemble_kernel<TY>, dim3(T, H), dim3(kLatentThreads), 0, stream, (TY*)q_out, (const TY*)q_abs, \
                               (const TY*)q, q_stride, H, nope, rank, rot_width, rot, cos_t, sin_t, max_pos, positions, T, err_flag)
    CVB_DISPATCH_DTYPE(dtype, CALL);
#undef CALL
    return launch_status();
}

extern "C" int cvb_latent_q_turn(void* q_out, const void* q, int T, int q_stride, int H, int nope, int rank, int rot_width, int rot,
                                 const float* cos_t, const float* sin_t, int max_pos, const int* positions, int dtype, int* err_flag,
                                 cudaStream_t stream) {
    if (T == 0 || rot_width == 0) return CVB_OK;
    if (T < 0 || H <= 0 || nope <= 0 || rank <= 0 || rot_width < 0 || max_pos <= 0) return CVB_E_SIZE;
    if (rot < 0 || rot > rot_width || rot % 2 || q_stride < H * (nope + rot_width)) return CVB_E_SHAPE;
    const int n16 = dtype == CVB_DTYPE_BF16 ? 8 : 4;
    const int64_t total = static_cast<int64_t>(T) * H * rot_width / n16;
    if (rot_width % n16 == 0 && rot % n16 == 0 && nope % n16 == 0 && rank % n16 == 0 && q_stride % n16 == 0 && total < (1 << 30) &&
        ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(q_out)) & 15) == 0) {
        const int64_t want = (total + 255) / 256;
        const unsigned blocks = static_cast<unsigned>(want < 148 * 8 ? want : 148 * 8);
#define CALL(TY) launch_kernel(latent_q_turn_vec_kernel<TY>, dim3(blocks), dim3(256), 0, stream, (TY*)q_out, (const TY*)q, q_stride, H, nope, rank, \
                               rot_width, rot, cos_t, sin_t, max_pos, positions, static_cast<int>(total), err_flag)
        CVB_DISPATCH_DTYPE(dtype, CALL);
#undef CALL
        return launch_status();
    }
    const int per_row = (H * rot_width + kLatentThreads - 1) / kLatentThreads;
#define CALL(TY) launch_kernel(latent_q_turn_kernel<TY>, dim3(T, per_row < 64 ? per_row : 64), dim3(kLatentThreads), 0, stream, (TY*)q_out, \
                               (const TY*)q, q_stride, H, nope, rank, rot_width, rot, cos_t, sin_t, max_pos, positions, err_flag)
    CVB_DISPATCH_DTYPE(dtype, CALL);
#undef CALL
    return launch_status();
}

extern "C" int cvb_head_gate(void* out, int out_stride, const void* o, const void* gate, int T, int gate_stride, int H, int vd, int per_element,
                             int dtype, cudaStream_t stream) {
    if (T == 0) return CVB_OK;
    if (T < 0 || H <= 0 || vd <= 0 || out_stride < H * vd || gate_stride < (per_element ? H * vd : H)) return CVB_E_SIZE;
    const int n16 = dtype == CVB_DTYPE_BF16 ? 8 : 4;
    const uintptr_t bases = reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(o) | (per_element ? reinterpret_cast<uintptr_t>(gate) : 0);
    const int64_t total = static_cast<int64_t>(T) * H * vd / n16;
    if (vd % n16 == 0 && out_stride % n16 == 0 && (!per_element || gate_stride % n16 == 0) && (bases & 15) == 0 && total < (1 << 30)) {
        const int64_t want = (total + 1023) / 1024;
        const unsigned blocks = static_cast<unsigned>(want < 148 * 8 ? want : 148 * 8);
#define CALL(TY) launch_kernel(head_gate_vec_kernel<TY>, dim3(blocks), dim3(256), 0, stream, (TY*)out, out_stride, (const TY*)o, (const TY*)gate, \
                               gate_stride, H, vd, T, per_element, static_cast<int>(total))
        CVB_DISPATCH_DTYPE(dtype, CALL);
#undef CALL
        return launch_status();
    }
    const int per_row = (H * vd + kLatentThreads - 1) / kLatentThreads;
#define CALL(TY) launch_kernel(head_gate_kernel<TY>, dim3(T, per_row < 64 ? per_row : 64), dim3(kLatentThreads), 0, stream, (TY*)out, out_stride, (const TY*)o, (const TY*)gate, \
                               gate_stride, H, vd, T, per_element)
    CVB_DISPATCH_DTYPE(dtype, CALL);
#undef CALL
    return launch_status();
}
