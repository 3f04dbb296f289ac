// kv_slab.cu — KV-cache slabs and the append (row quantise-on-write) kernels.
//
// Layout: one arena per cache, holding 2*n_layers slabs (K then V per layer), each slab starting
// on a 1024-byte boundary.  Inside a slab rows are head-major, ggml view [hd, max_ctx, n_kv, n_streams]:
//   nb1 = row bytes (hd*2 for F16, hd/32*34 for Q8_0), nb2 = ctx_rows*nb1, nb3 = n_kv*nb2,
// with ctx_rows = max_ctx rounded up to a multiple of 32 so that every head's row range starts on a
// 16-byte boundary for both row sizes (a Q8_0 row of head_dim 128 is 136 bytes).
#include <cstdio>
#include <new>

#include "fattn_common.cuh"

struct b200_kv_cache {
    b200_kv_config cfg;
    uint8_t* arena;   // cudaMalloc'ed
    uint8_t* base;    // arena rounded up to 1024
    size_t slab_bytes;
    size_t row_bytes;
    int64_t ctx_rows;
    int device;
};

namespace b200 {
namespace {

// Rows of K and V in one launch: a warp takes 256 floats at a time (two rows of head_dim 128, four of 64), eight per
// thread.  The operation is bound by its bytes (4 B in, 1.06 or 2 B out per element) when many rows enter, by
// the launch when one does; what the first form (one thread per pair or element, three 64-bit divisions each, 16-bit
// stores, a launch each for K and V) spent its time on was index arithmetic: 407 rows x 64 heads of head_dim 128 into
// Q8_0 66 us, this one 9.7 us, against 5.2 us of memory time (F16 7.7 us; 1500 rows 28 and 22 us: 4.4 and 6.6 TB/s; what
// Q8_0 adds is the arithmetic of its blocks).  One row per head: two launches of 2.8 us -> one of 2.0, on which the
// attention behind it waits (its set-up runs meanwhile).
struct AppendArgs {
    const uint8_t* src[2];                   // K, V
    int64_t snb1[2], snb2[2], snb3[2];
    uint8_t* dst[2];
    int64_t dnb1, dnb2, dnb3;                // K and V slabs have one geometry
    int n_new[2];
    int hd, n_kv, chunks, ctx_rows, pos0;    // chunks: CTAs per (stream, head)
    const int32_t* pos;
};

// Four consecutive floats; V16: 16-byte aligned rows (8-byte alignment is what the entry point asks for).
template <bool V16>
__device__ __forceinline__ float4 load4(const uint8_t* p) {
    if (V16) return __ldcs(reinterpret_cast<const float4*>(p));
    const float2 a = __ldcs(reinterpret_cast<const float2*>(p)), b = __ldcs(reinterpret_cast<const float2*>(p + 8));
    return make_float4(a.x, a.y, b.x, b.y);
}

// (int)roundf(t) for |t| < 2^22 without either unit's conversions: |t| + 1/2 truncated to an integer by two additions that
// round towards zero (the first cannot reach an integer the exact sum does not reach), then the sign; NaN gives 0.  In a block
// of values below 4e-37 1/d is beyond a float and t infinite: the low byte is that of the saturated conversion, 0xFF for
// +inf, 0 for -inf (a branch for such blocks cost 0.2 us per launch).
__device__ __forceinline__ uint32_t round_away(float t) {
    asm("min.NaN.f32 %0, %0, 0f437F0000;" : "+f"(t));   // 255; a NaN stays one
    const float m = fmaxf(fabsf(t), 0.0f);
    const int32_t k = __float_as_int(__fadd_rz(__fadd_rz(m, 0.5f), 8388608.0f)), sign = __float_as_int(t) >> 31;
    return (uint32_t)((k ^ sign) - sign);
}
// Low bytes of four words.
__device__ __forceinline__ uint32_t low_bytes(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

// Q8_0 blocks, bit-identical to gguf-py quantize_blocks: d = amax/127 (fp32), stored as fp16; q = roundf(x * (1/d)) with
// 1/d = 0 for d == 0.  Four lanes share a block, eight elements each.
// A block is 34 bytes.  In a row of an even number of blocks (head_dim 64 / 128: rows start on a 4-byte boundary) the
// quants of the odd blocks fill aligned words and those of the even ones straddle them by two bytes; there a lane takes
// the upper half of its left neighbour's last word (the first lane the scale) and the row leaves in 32-bit stores.
template <bool Q8, bool V16, int U>
__global__ void __launch_bounds__(256) kv_append_kernel(const AppendArgs a) {
    // launched with programmatic stream serialisation: the attention of this layer may set itself up meanwhile; rows are read and
    // written behind the wait, when the previous kernel of the stream has completed
    let_dependents_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lpr = a.hd / 8, rpw = 32 / lpr;   // lanes per row (4, 8, 12, 16); rows per warp instruction
    const int sub = lane / lpr, c = (lane - sub * lpr) * 8;
    const int which = blockIdx.y, sh = blockIdx.x / a.chunks, chunk = blockIdx.x - sh * a.chunks, s = sh / a.n_kv, h = sh - s * a.n_kv;
    const int n_new = a.n_new[which];
    // A warp's first rows (all it has where one token per stream enters) are brought into L2 while the previous kernel still runs.  Rows that
    // are not there yet cost a trip to memory on the chain of a decode step otherwise: 32 streams of an F16 cache, 30 layers, 470 ->
    // 458 us; 20 streams, 20 layers, 157 -> 148.  A few rows per stream gain as much, in one wave of CTAs or several (the append alone,
    // 16 streams of 4 rows 1.7 -> 1.45 us, 256 of 8 6.8 -> 5.7, 64 of 30 6.1 -> 5.3).  The form of
    // two rows in flight per warp was not measured with it.
    if (U == 1) {
        const int row = (chunk * (blockDim.x >> 5) + warp) * rpw + sub;
        if (sub < rpw && row < n_new && (c & 31) == 0)
            prefetch_l2(a.src[which] + (int64_t)h * a.snb2[which] + (int64_t)s * a.snb3[which] + (int64_t)row * a.snb1[which] + c * 4);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int p0 = a.pos ? a.pos[s] : a.pos0;
    const int row_lo = max(0, -p0), row_hi = sub < rpw ? min(n_new, a.ctx_rows - p0) : 0;   // out-of-range rows are dropped, never written
    const uint8_t* src = a.src[which] + (int64_t)h * a.snb2[which] + (int64_t)s * a.snb3[which] + (int64_t)c * 4;
    uint8_t* dst = a.dst[which] + (int64_t)h * a.dnb2 + (int64_t)s * a.dnb3 + (int64_t)p0 * a.dnb1;
    const int step = a.chunks * (blockDim.x >> 5) * rpw;
    for (int row0 = (chunk * (blockDim.x >> 5) + warp) * rpw; row0 < n_new; row0 += U * step) {
        float4 x[U][2];
        bool live[U];
#pragma unroll
        for (int u = 0; u < U; u++) {   // the loads of U rows in flight
            const int row = row0 + u * step + sub;
            live[u] = row >= row_lo && row < row_hi;
            x[u][0] = x[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live[u]) {
                const uint8_t* p = src + (int64_t)row * a.snb1[which];
                x[u][0] = load4<V16>(p), x[u][1] = load4<V16>(p + 16);
            }
        }
        // The rows of the next turn into L2 meanwhile: 16 x 407 rows of 8 heads into F16 15.5 -> 14.5 us, 8 x 1500 27.1 -> 26.0.  (Into Q8_0, whose
        // arithmetic covers the loads, 1 %, and the attention behind 8 x 407 rows then starts 0.3 us later.)
        if (U > 1 && !Q8) {
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int row = row0 + (U + u) * step + sub;
                if (row < row_hi && (c & 31) == 0) prefetch_l2(src + (int64_t)row * a.snb1[which]);
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            uint8_t* row_out = dst + (int64_t)(row0 + u * step + sub) * a.dnb1;
            const float f[8] = {x[u][0].x, x[u][0].y, x[u][0].z, x[u][0].w, x[u][1].x, x[u][1].y, x[u][1].z, x[u][1].w};
            if (!Q8) {
                if (live[u])
                    *reinterpret_cast<uint4*>(row_out + c * 2) =
                        make_uint4(pack_half2(f[0], f[1]), pack_half2(f[2], f[3]), pack_half2(f[4], f[5]), pack_half2(f[6], f[7]));
                continue;
            }
            float amax = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; i++) amax = fmaxf(amax, fabsf(f[i]));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
            const float d = __fdiv_rn(amax, 127.0f);
            const float id = d != 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
            uint32_t q[8];
#pragma unroll
            for (int i = 0; i < 8; i++) q[i] = round_away(__fmul_rn(f[i], id));
            const uint32_t w0 = low_bytes(q[0], q[1], q[2], q[3]), w1 = low_bytes(q[4], q[5], q[6], q[7]);
            const uint32_t dbits = __half_as_ushort(__float2half_rn(d));
            const uint32_t left = __shfl_up_sync(0xffffffffu, w1, 1);
            if (!live[u]) continue;
            const int blk = c >> 5, i = (c & 31) >> 3;   // lane i of the block's four
            uint8_t* out = row_out + blk * 34 + 8 * i;
            if ((a.hd & 63) == 0) {
                if (blk & 1) {
                    *reinterpret_cast<uint32_t*>(out + 2) = w0;
                    *reinterpret_cast<uint32_t*>(out + 6) = w1;
                    if (i == 0) *reinterpret_cast<uint16_t*>(out) = (uint16_t)dbits;
                } else {
                    *reinterpret_cast<uint32_t*>(out) = (w0 << 16) | (i == 0 ? dbits : left >> 16);
                    *reinterpret_cast<uint32_t*>(out + 4) = __funnelshift_l(w0, w1, 16);
                    if (i == 3) *reinterpret_cast<uint16_t*>(out + 8) = (uint16_t)(w1 >> 16);
                }
            } else {   // an odd number of blocks: rows are only 2-byte aligned
                *reinterpret_cast<uint16_t*>(out + 2) = (uint16_t)w0;
                *reinterpret_cast<uint16_t*>(out + 4) = (uint16_t)(w0 >> 16);
                *reinterpret_cast<uint16_t*>(out + 6) = (uint16_t)w1;
                *reinterpret_cast<uint16_t*>(out + 8) = (uint16_t)(w1 >> 16);
                if (i == 0) *reinterpret_cast<uint16_t*>(out) = (uint16_t)dbits;
            }
        }
    }
}

template <bool Q8, bool V16>
cudaError_t launch_append(AppendArgs a, int n_heads_total, cudaStream_t st) {
    // One token per stream: a warp per (stream, head).  Many rows: eight warps per CTA, four rows (of 128) in flight per warp, and
    // no more CTAs than are resident at once (six per SM), so that a warp's next rows are requested without a new CTA's start.
    const int rpw = 32 / (a.hd / 8), n_new = a.n_new[0] > a.n_new[1] ? a.n_new[0] : a.n_new[1];
    const int units = (n_new + rpw - 1) / rpw;   // warp instructions per (stream, head)
    const int u = units >= 16 ? 2 : 1, warps = (units + u - 1) / u, per_block = warps < 8 ? warps : 8;
    const int full = (warps + per_block - 1) / per_block, resident = (148 * 6 + 2 * n_heads_total - 1) / (2 * n_heads_total);
    a.chunks = full < resident ? full : resident;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.chunks * n_heads_total, 2);
    cfg.blockDim = dim3(32 * per_block);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return u == 2 ? cudaLaunchKernelEx(&cfg, kv_append_kernel<Q8, V16, 2>, a) : cudaLaunchKernelEx(&cfg, kv_append_kernel<Q8, V16, 1>, a);
}

}  // namespace
}  // namespace b200

extern "C" {

B200_API int b200_kv_create(const b200_kv_config* cfg, b200_kv_cache** out) {
    if (!cfg || !out) return B200_E_NULL;
    *out = nullptr;
    if (cfg->type != B200_TYPE_F16 && cfg->type != B200_TYPE_Q8_0) return B200_E_TYPE;
    if (cfg->head_dim <= 0 || cfg->head_dim % 32 || cfg->head_dim > 128) return B200_E_UNSUPPORTED;
    if (cfg->n_kv_heads <= 0 || cfg->n_layers <= 0 || cfg->max_ctx <= 0 || cfg->n_streams <= 0) return B200_E_SHAPE;
    b200_kv_cache* kv = new (std::nothrow) b200_kv_cache();
    if (!kv) return B200_E_CUDA;
    kv->cfg = *cfg;
    kv->row_bytes = cfg->type == B200_TYPE_F16 ? (size_t)cfg->head_dim * 2 : (size_t)cfg->head_dim / 32 * 34;
    kv->ctx_rows = ((int64_t)cfg->max_ctx + 31) / 32 * 32;
    const size_t raw = kv->row_bytes * kv->ctx_rows * cfg->n_kv_heads * cfg->n_streams;
    kv->slab_bytes = (raw + 1023) / 1024 * 1024;
    const size_t total = kv->slab_bytes * 2 * cfg->n_layers + 1024;
    if (cudaGetDevice(&kv->device) != cudaSuccess) {
        delete kv;
        return B200_E_NO_DEVICE;
    }
    if (cudaMalloc((void**)&kv->arena, total) != cudaSuccess) {
        cudaGetLastError();
        delete kv;
        return B200_E_CUDA;
    }
    kv->base = (uint8_t*)(((uintptr_t)kv->arena + 1023) / 1024 * 1024);
    // a cleared cache reads as zeros (whisper clears kv_pad at init, src/crispasr.cpp:1506)
    if (cudaMemset(kv->arena, 0, total) != cudaSuccess) {
        cudaFree(kv->arena);
        delete kv;
        return B200_E_CUDA;
    }
    *out = kv;
    return B200_OK;
}

B200_API void b200_kv_destroy(b200_kv_cache* kv) {
    if (!kv) return;
    if (kv->arena) cudaFree(kv->arena);
    delete kv;
}

B200_API size_t b200_kv_bytes(const b200_kv_cache* kv) { return kv ? kv->slab_bytes * 2 * kv->cfg.n_layers : 0; }

B200_API int b200_kv_view(const b200_kv_cache* kv, int layer, int64_t n_rows, b200_tensor* k, b200_tensor* v) {
    if (!kv || !k || !v) return B200_E_NULL;
    if (layer < 0 || layer >= kv->cfg.n_layers || n_rows <= 0 || n_rows > kv->ctx_rows) return B200_E_SHAPE;
    for (int which = 0; which < 2; which++) {
        b200_tensor* t = which ? v : k;
        t->data = kv->base + kv->slab_bytes * (2 * (size_t)layer + which);
        t->type = kv->cfg.type;
        t->reserved = 0;
        t->ne[0] = kv->cfg.head_dim, t->ne[1] = n_rows, t->ne[2] = kv->cfg.n_kv_heads, t->ne[3] = kv->cfg.n_streams;
        t->nb[0] = kv->cfg.type == B200_TYPE_F16 ? 2 : 34;
        t->nb[1] = kv->row_bytes;
        t->nb[2] = kv->row_bytes * kv->ctx_rows;
        t->nb[3] = t->nb[2] * kv->cfg.n_kv_heads;
    }
    return B200_OK;
}

B200_API int b200_kv_append(b200_kv_cache* kv, int layer, const b200_tensor* k_new, const b200_tensor* v_new,
                            const int32_t* pos, int32_t pos0, void* cuda_stream) {
    if (!kv || !k_new || !v_new) return B200_E_NULL;
    if (layer < 0 || layer >= kv->cfg.n_layers) return B200_E_SHAPE;
    b200_tensor kd, vd;
    b200_kv_view(kv, layer, kv->ctx_rows, &kd, &vd);
    b200::AppendArgs a = {};
    bool v16 = true;
    for (int which = 0; which < 2; which++) {
        const b200_tensor* s = which ? v_new : k_new;
        if (!s->data) return B200_E_NULL;
        if (s->type != B200_TYPE_F32) return B200_E_TYPE;
        if (s->nb[0] != 4) return B200_E_STRIDE;
        if ((uintptr_t)s->data % 8 || s->nb[1] % 8 || s->nb[2] % 8 || s->nb[3] % 8) return B200_E_ALIGN;
        if (s->ne[0] != kv->cfg.head_dim || s->ne[2] != kv->cfg.n_kv_heads || s->ne[3] != kv->cfg.n_streams)
            return B200_E_SHAPE;
        if (s->ne[1] <= 0 || s->ne[1] > kv->ctx_rows) return B200_E_SHAPE;
        if (!pos && (pos0 < 0 || pos0 + s->ne[1] > kv->ctx_rows)) return B200_E_SHAPE;
        a.src[which] = (const uint8_t*)s->data;
        a.snb1[which] = (int64_t)s->nb[1], a.snb2[which] = (int64_t)s->nb[2], a.snb3[which] = (int64_t)s->nb[3];
        a.n_new[which] = (int)s->ne[1];
        a.dst[which] = (uint8_t*)(which ? vd : kd).data;
        v16 = v16 && (uintptr_t)s->data % 16 == 0 && s->nb[1] % 16 == 0 && s->nb[2] % 16 == 0 && s->nb[3] % 16 == 0;
    }
    a.dnb1 = (int64_t)kd.nb[1], a.dnb2 = (int64_t)kd.nb[2], a.dnb3 = (int64_t)kd.nb[3];
    a.hd = kv->cfg.head_dim, a.n_kv = kv->cfg.n_kv_heads;
    a.ctx_rows = (int)kv->ctx_rows, a.pos = pos, a.pos0 = pos0;
    cudaStream_t st = (cudaStream_t)cuda_stream;
    const int n = kv->cfg.n_kv_heads * kv->cfg.n_streams;
    const bool q8 = kv->cfg.type == B200_TYPE_Q8_0;
    const cudaError_t e = q8 ? (v16 ? b200::launch_append<true, true>(a, n, st) : b200::launch_append<true, false>(a, n, st))
                             : (v16 ? b200::launch_append<false, true>(a, n, st) : b200::launch_append<false, false>(a, n, st));
    if (e != cudaSuccess || cudaGetLastError() != cudaSuccess) return B200_E_CUDA;
    return B200_OK;
}

B200_API int b200_kv_copy_stream(b200_kv_cache* kv, int dst_stream, int src_stream, int64_t n_rows, void* cuda_stream) {
    if (!kv) return B200_E_NULL;
    if (dst_stream < 0 || src_stream < 0 || dst_stream >= kv->cfg.n_streams || src_stream >= kv->cfg.n_streams)
        return B200_E_SHAPE;
    if (n_rows < 0 || n_rows > kv->ctx_rows) return B200_E_SHAPE;
    if (dst_stream == src_stream || n_rows == 0) return B200_OK;
    const size_t head_pitch = kv->row_bytes * kv->ctx_rows;
    const size_t stream_pitch = head_pitch * kv->cfg.n_kv_heads;
    for (int slab = 0; slab < 2 * kv->cfg.n_layers; slab++) {
        uint8_t* base = kv->base + kv->slab_bytes * slab;
        // one 2-D copy per slab: n_kv_heads rows of n_rows*row_bytes bytes, head_pitch apart
        if (cudaMemcpy2DAsync(base + stream_pitch * dst_stream, head_pitch, base + stream_pitch * src_stream, head_pitch,
                              (size_t)n_rows * kv->row_bytes, kv->cfg.n_kv_heads, cudaMemcpyDeviceToDevice,
                              (cudaStream_t)cuda_stream) != cudaSuccess) {
            cudaGetLastError();
            return B200_E_CUDA;
        }
    }
    return B200_OK;
}

}  // extern "C"
