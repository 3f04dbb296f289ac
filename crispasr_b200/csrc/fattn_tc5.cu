// fattn_tc5.cu — prefill attention on the Blackwell tensor path: TMA-staged K/V tiles, tcgen05.mma
// with accumulators in tensor memory (TMEM), fp32 online softmax by one thread per query row.
//
// One CTA = one 128-row query tile of one (head, batch entry); 192 threads:
//   warps 0-3  softmax / correction / epilogue: thread r owns query row r (TMEM lane r)
//   warp  4    TMA producer (one lane): K and V tiles of 128 keys, 128-byte swizzled
//   warp  5    TMEM allocator and the single tcgen05.mma issuing thread
// TMEM (256 columns per CTA, so two CTAs share an SM and fill each other's softmax bubbles):
//   cols [0,128)       S = Q.K^T tile, fp32            (128 lanes x 128 keys)
//   cols [0,64)        P = exp2(S - m), f16x2 packed    (aliases S once the row has been read)
//   cols [128,128+HD)  O accumulator, fp32
// Shared memory: Q tile (written once by the softmax warps, converted to f16, swizzled by hand so
// both F32 and F16 Q with any strides work), NSTG K tiles and NSTG V tiles (TMA, SWIZZLE_128B).
// Per KV tile: S = Q.K^T (SS MMA, both operands K-major) -> softmax threads read S, write P to TMEM
// -> O += P.V (TS MMA: A = P from TMEM, B = V from shared memory, MN-major).
// The rescale of O by exp2(m_old - m_new) is lazy: it only happens when a row's maximum grew by
// more than 2^8, so P stays within f16 range and the common case touches O only in the MMA.
//
// Every mbarrier wait is bounded: when a wait runs out the CTA raises a flag, all roles leave their
// loops, in-flight copies are drained (bounded), TMEM is released and a device status word is set.
#include <cuda.h>

#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "fattn_tc5.cuh"

namespace b200 {

__device__ int g_tc5_status = 0;  // 0 ok, 1 = a bounded wait ran out in some CTA

namespace {

constexpr int kTile = 128;              // query rows per CTA and keys per step
constexpr int kPanelBytes = 128 * 128;  // 128 rows x 64 f16
constexpr int kThreadsTc5 = 192;
constexpr uint32_t kTmemCols = 256;
constexpr uint32_t kWaitLimit = 1u << 22;
constexpr float kRescaleThreshold = 8.0f;  // log2 units: P <= 256 stays well inside f16 range

// ---- PTX wrappers -----------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Non-blocking test.  The answer takes about 120 clocks to come back even when the phase completed long ago, so a
// wait whose barrier is normally complete is probed early (the result is consumed after other work) and only falls
// back to the polling wait when the probe said no.
__device__ __forceinline__ uint32_t mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok;
}
// Bounded wait. Returns false when the CTA is aborting (this wait or another one ran out).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    for (uint32_t it = 0; it < kWaitLimit; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if (it > 256) {
            if (*abort_flag) return false;
            __nanosleep(64);
        }
    }
    *abort_flag = 1;
    atomicExch(&g_tc5_status, 1);
    return false;
}
// One answer for all lanes: the issuing warps elect a lane behind their waits, which needs every lane there, also when a wait
// ran out for some.
__device__ __forceinline__ bool warp_all(bool ok) { return __all_sync(0xffffffffu, ok); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2,
                                            int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}

// The box of such a load into L2 only, with no copy to shared memory.
__device__ __forceinline__ void tma_prefetch_4d(const CUtensorMap* map, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];"
                 ::"l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
                 : "memory");
}

// Tensor store shared -> global as its own bulk group; the caller waits for the group's reads of shared memory
// before the CTA ends.  The innermost coordinate times the element size must be a multiple of 16 bytes, and no
// coordinate may be negative.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                 ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
                 : "memory");
}
__device__ __forceinline__ void tma_store_commit_and_wait_read() {
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

// Shared-memory matrix descriptor, SWIZZLE_128B, descriptor version 1 (sm_100).
//   K-major operand : rows of 128 bytes, 8-row groups 1024 bytes apart  -> LBO = 16 B (unused), SBO = 1024 B
//   MN-major operand: 64-element chunks `lbo` bytes apart, 8-k groups 1024 bytes apart
// The two 32-bit words of a descriptor.  Only the low word carries the address (bits 0-13, in 16-byte units),
// so stepping through an operand is one 32-bit add: the issuing thread's instruction latency, not the tensor
// pipe, bounds how fast small MMAs can be issued.
__device__ __forceinline__ uint32_t smem_desc_lo(uint32_t addr, uint32_t lbo_bytes) {
    return ((addr & 0x3FFFFu) >> 4) | (((lbo_bytes >> 4) & 0x3FFFu) << 16);
}
__device__ __forceinline__ constexpr uint32_t smem_desc_hi(uint32_t sbo_bytes) {
    return ((sbo_bytes >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29);
}
__device__ __forceinline__ uint64_t desc64(uint32_t lo, uint32_t hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
    return d;
}

// Instruction descriptor for kind::f16: F16 A/B, F32 accumulate, M = 128.
__host__ __device__ constexpr uint32_t idesc_f16(int n, bool b_mn_major) {
    return (1u << 4) | (0u << 7) | (0u << 10) | (0u << 15) | ((b_mn_major ? 1u : 0u) << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTile >> 4) << 24);
}

__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc)
        : "memory");
}
// One lane of a converged warp.  The issuing warps run their loops with all lanes and put only the tensor instructions
// behind this: descriptors and TMEM addresses of a warp-uniform loop live in uniform registers, which is where
// tcgen05.mma reads them.  Behind `if (lane == 0)` the compiler cannot know the loop to be uniform and moves every operand
// over per instruction; the issue chain between P and the next score tile is what the softmax warps wait for (64 windows
// of the large encoder 1139 -> 956 us by this alone).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
          "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
          "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Packed fp32 pairs (one issue slot for two lanes of work on sm_100) and the three-input maximum.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// What a row without a finite reference subtracts: any finite score gives P = +inf, which the row's sum shows, however far
// below 0 the score lies (against 0 a row of scores below -126 would underflow unseen); a score of -inf still gives 0.
constexpr float kNoReference = -1e30f;
// Sum of a row over a step's 64 keys (rel-pos kernel: over half of a tile's 128) above which the reference is taken anew from
// the maximum.  Not a question of range (f16 holds P up to 2^16) but of precision: a key that carries the row has P = 1, exact
// in f16, only if it is the reference itself.  64 equal scores sum to 64, so the bound lies above that; random scores of unit
// variance stay below 30 (a bound of 32 redoes most steps: 1230 us at 64 windows).  Error against 64 bits (relative 2-norm, in
// brackets that of a maximum kept within 2^8, and of a bound of 2^12 with a reference from 16 scores): variance 1, 1500 keys
// 2.063e-4 (2.063e-4, 2.068e-4), variance 4, 700 keys 1.88e-4 (1.97e-4, 2.05e-4), variance 64 1.16e-4 (1.18e-4, 1.59e-4).
constexpr float kRedoSum = 96.0f, kRedoSumRelpos = 256.0f;

// x bounded to [-126, 126]; a NaN stays one (fmaxf and fminf would drop it).
__device__ __forceinline__ float clamp126(float x) {
    float y;
    asm("max.NaN.f32 %0, %1, 0fC2FC0000;\n\tmin.NaN.f32 %0, %0, 0f42FC0000;" : "=f"(y) : "f"(x));
    return y;
}
// 2^t of a pair on the FMA pipe: t = n + f with |f| <= 1/2 (adding 1.5 * 2^23 rounds and leaves n in the low bits), a
// degree-4 minimax polynomial of 2^f (computed here by weighted least squares; relative error 2.7e-6, a hundredth of the
// rounding of P to f16), times 2^n (which keeps a NaN, where adding n to the exponent field would not).  Any t may come:
// against a reference that is far below the score t has no bound, and the caller finds that out from the sum of the
// results.  t below -126 gives 2^-126 (0 as f16), t above 126 gives 2^126: an exponent field that ran over would be a small
// negative number, which no sum shows.
__device__ __forceinline__ void poly_ex2(float t0, float t1, float& p0, float& p1) {
    const uint64_t magic = pack2(12582912.0f, 12582912.0f), nmagic = pack2(-12582912.0f, -12582912.0f), neg1 = pack2(-1.0f, -1.0f);
    const uint64_t x = pack2(clamp126(t0), clamp126(t1)), r = add2(x, magic), n = add2(r, nmagic), f = fma2(n, neg1, x);
    const float C0 = 0.9999992847442627f, C1 = 0.6931217908859253f, C2 = 0.240247443318367f, C3 = 0.05591785907745361f, C4 = 0.009570102207362652f;
    uint64_t p = fma2(f, pack2(C4, C4), pack2(C3, C3));
    p = fma2(p, f, pack2(C2, C2));
    p = fma2(p, f, pack2(C1, C1));
    p = fma2(p, f, pack2(C0, C0));
    float ra, rb;
    unpack2(r, ra, rb);
    const float e0 = __uint_as_float((__float_as_uint(ra) << 23) + 0x3F800000u), e1 = __uint_as_float((__float_as_uint(rb) << 23) + 0x3F800000u);   // 2^n
    unpack2(mul2(p, pack2(e0, e1)), p0, p1);
}

// Eight Q elements [c0, c0+8) of one row as packed f16 (F32 rows are rounded to nearest even).
__device__ __forceinline__ uint4 q_chunk(const uint8_t* rowp, int type, int c0, bool vec16) {
    uint4 out;
    if (type == B200_TYPE_F16) {
        if (vec16) return load_global(reinterpret_cast<const uint4*>(rowp + 2 * c0));
        const uint16_t* h = reinterpret_cast<const uint16_t*>(rowp + 2 * c0);
        out.x = h[0] | ((uint32_t)h[1] << 16), out.y = h[2] | ((uint32_t)h[3] << 16);
        out.z = h[4] | ((uint32_t)h[5] << 16), out.w = h[6] | ((uint32_t)h[7] << 16);
        return out;
    }
    float f[8];
    if (vec16) {
        const float4 a = load_global(reinterpret_cast<const float4*>(rowp + 4 * c0));
        const float4 b = load_global(reinterpret_cast<const float4*>(rowp + 4 * c0 + 16));
        f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w, f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) f[i] = *reinterpret_cast<const float*>(rowp + 4 * (c0 + i));
    }
    out.x = pack_half2(f[0], f[1]), out.y = pack_half2(f[2], f[3]);
    out.z = pack_half2(f[4], f[5]), out.w = pack_half2(f[6], f[7]);
    return out;
}

// {hi, lo} -> packed f16x2 with lo in the low half
__device__ __forceinline__ uint32_t cvt_f16x2(float lo, float hi) {
    uint32_t y;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(y) : "f"(hi), "f"(lo));
    return y;
}
// Maximum of 64 score columns held in two 32-register chunks; columns >= n_valid (tile-relative) are skipped.
__device__ __forceinline__ float row_max64(const uint32_t (&sreg)[2][32], int col0, int n_valid) {
    float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int q2 = 0; q2 < 2; q2++)
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
            const float s0 = (col0 + q2 * 32 + i < n_valid) ? __uint_as_float(sreg[q2][i]) : -INFINITY;
            const float s1 = (col0 + q2 * 32 + i + 1 < n_valid) ? __uint_as_float(sreg[q2][i + 1]) : -INFINITY;
            mx[(i >> 1) & 3] = max3(mx[(i >> 1) & 3], s0, s1);
        }
    return max3(fmaxf(mx[0], mx[1]), mx[2], mx[3]);
}

// 32 score columns -> 16 packed f16x2 probabilities exp2(s*c - m).  Per pair of columns: one three-input maximum, one packed
// FMA, two ex2, one packed add, one f16x2 convert.  The accumulators are kept by the caller (mx[8], ls[4] live across the
// four chunks of a tile), which lets the TMEM load of a later chunk run under the exponentials of an earlier one.
__device__ __forceinline__ void softmax32(const uint32_t (&sreg)[32], uint32_t* preg16, uint64_t c2, uint64_t nm2, float (&mx)[8], uint64_t (&ls)[4]) {
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        const float s0 = __uint_as_float(sreg[i]), s1 = __uint_as_float(sreg[i + 1]);
        mx[(i >> 1) & 7] = max3(mx[(i >> 1) & 7], s0, s1);
        float t0, t1;
        unpack2(fma2(pack2(s0, s1), c2, nm2), t0, t1);
        const float p0 = ex2(t0), p1 = ex2(t1);
        ls[(i >> 1) & 3] = add2(ls[(i >> 1) & 3], pack2(p0, p1));
        preg16[i >> 1] = cvt_f16x2(p0, p1);
    }
}

// 64 consecutive F16 mask values starting at `mptr` as eight 16-byte loads, all in flight at once (2-byte loads
// where the address is not 16-byte aligned); values at or beyond `avail` (the end of the mask row) read as 0 and
// are never touched in memory.
__device__ __forceinline__ void load_mask64(uint4 (&mv)[8], const uint8_t* mptr, int avail) {
#pragma unroll
    for (int q = 0; q < 8; q++) {
        if (q * 8 + 8 <= avail && ((reinterpret_cast<uintptr_t>(mptr) & 15) == 0)) {
            mv[q] = load_behind_wait(reinterpret_cast<const uint4*>(mptr + q * 16));
        } else {   // the end of the row, or a row that does not start on a 16-byte boundary (mask rows hold exactly Lk values)
            uint16_t hv[8];
#pragma unroll
            for (int i = 0; i < 8; i++)
                hv[i] = (q * 8 + i < avail) ? load_behind_wait(reinterpret_cast<const uint16_t*>(mptr + (q * 8 + i) * 2)) : (uint16_t)0;
            mv[q] = make_uint4(hv[0] | ((uint32_t)hv[1] << 16), hv[2] | ((uint32_t)hv[3] << 16), hv[4] | ((uint32_t)hv[5] << 16),
                               hv[6] | ((uint32_t)hv[7] << 16));
        }
    }
}
// Mask value pair (columns i, i+1 of the 64, i even) of a block loaded by load_mask64.
__device__ __forceinline__ float2 mask_pair(const uint4 (&mv)[8], int i) {
    const uint4& v = mv[i >> 3];
    const int u = (i & 7) >> 1;
    const uint32_t w = u == 0 ? v.x : (u == 1 ? v.y : (u == 2 ? v.z : v.w));
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
}

// Explicit F16 mask: turns 64 raw scores into log2-domain logits t = s*c + mask*log2(e) in place (mask -inf stays
// -inf).  `mptr` points at the mask value of the first of the 64 columns, `avail` is how many mask columns exist
// from there to the end of the mask row (loads never go past it).
__device__ __forceinline__ void apply_mask64(uint32_t (&sreg)[2][32], const uint8_t* mptr, int avail, float c) {
    uint4 mv[8];
    load_mask64(mv, mptr, avail);
#pragma unroll
    for (int i = 0; i < 64; i += 2) {
        const float2 m2 = mask_pair(mv, i);
        sreg[i >> 5][i & 31] = __float_as_uint(fmaf(__uint_as_float(sreg[i >> 5][i & 31]), c, m2.x * kLog2e));
        sreg[i >> 5][(i + 1) & 31] = __float_as_uint(fmaf(__uint_as_float(sreg[i >> 5][(i + 1) & 31]), c, m2.y * kLog2e));
    }
}

// Explicit mask, fused form: 64 raw scores and their 64 mask values -> probabilities in one pass,
// x = s*c + (mask*log2(e) - m) with two packed FMAs per pair (folding the mask into the scores first and subtracting the
// maximum afterwards costs four scalar operations more per pair, and this path is bound by instruction issue).  The
// running maximum is tracked on x; the caller adds m back.  Columns >= n_valid (tile-relative) are dead.
template <bool MASKED>
__device__ __forceinline__ void softmax64_masked(const uint32_t (&sreg)[2][32], const uint4 (&mv)[8], uint32_t (&preg)[32], float c,
                                                 float m_use, int col0, int n_valid, float& mx_io, float& lsum_io) {
    float mx[8];
    uint64_t ls[4] = {0ull, 0ull, 0ull, 0ull};
    const uint64_t c2 = pack2(c, c), l2e2 = pack2(kLog2e, kLog2e), nm2 = pack2(-m_use, -m_use);
#pragma unroll
    for (int i = 0; i < 8; i++) mx[i] = -INFINITY;
#pragma unroll
    for (int i = 0; i < 64; i += 2) {
        const float2 m2 = mask_pair(mv, i);
        float x0, x1;
        unpack2(fma2(pack2(__uint_as_float(sreg[i >> 5][i & 31]), __uint_as_float(sreg[i >> 5][(i + 1) & 31])), c2,
                     fma2(pack2(m2.x, m2.y), l2e2, nm2)), x0, x1);
        if (MASKED) {
            if (col0 + i >= n_valid) x0 = -INFINITY;
            if (col0 + i + 1 >= n_valid) x1 = -INFINITY;
        }
        mx[(i >> 1) & 7] = max3(mx[(i >> 1) & 7], x0, x1);
        const float p0 = ex2(x0), p1 = ex2(x1);
        ls[(i >> 1) & 3] = add2(ls[(i >> 1) & 3], pack2(p0, p1));
        preg[i >> 1] = cvt_f16x2(p0, p1);
    }
    mx_io = max3(mx_io, max3(fmaxf(mx[0], mx[1]), mx[2], mx[3]), max3(fmaxf(mx[4], mx[5]), mx[6], mx[7]));
    float l0, l1;
    unpack2(add2(add2(ls[0], ls[1]), add2(ls[2], ls[3])), l0, l1);
    lsum_io += l0 + l1;
}

// One query row (HD elements) -> f16, written into the 128-byte swizzled operand tile: row r, 16-byte chunk c of
// panel p at p*16384 + r*128 + ((c ^ (r & 7)) * 16).  The type is tested once and all loads of the row are issued
// before the first store, so the row costs one memory round trip instead of HD/8.
template <int HD>
__device__ __forceinline__ void load_q_row(uint8_t* tile, int r, const uint8_t* rowp, int type, bool vec16, bool valid) {
    uint4 v[HD / 8];
    if (!valid) {
#pragma unroll
        for (int c = 0; c < HD / 8; c++) v[c] = make_uint4(0u, 0u, 0u, 0u);
    } else if (type == B200_TYPE_F16 && vec16) {
#pragma unroll
        for (int c = 0; c < HD / 8; c++) v[c] = load_global(reinterpret_cast<const uint4*>(rowp) + c);
    } else if (type == B200_TYPE_F32 && vec16) {
#pragma unroll
        for (int c0 = 0; c0 < HD / 8; c0 += 4) {  // 4 chunks = 8 float4 in flight
            float4 f[8];
#pragma unroll
            for (int i = 0; i < 8; i++) f[i] = load_global(reinterpret_cast<const float4*>(rowp) + c0 * 2 + i);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                v[c0 + i].x = pack_half2(f[2 * i].x, f[2 * i].y), v[c0 + i].y = pack_half2(f[2 * i].z, f[2 * i].w);
                v[c0 + i].z = pack_half2(f[2 * i + 1].x, f[2 * i + 1].y), v[c0 + i].w = pack_half2(f[2 * i + 1].z, f[2 * i + 1].w);
            }
        }
    } else {
#pragma unroll
        for (int c = 0; c < HD / 8; c++) v[c] = q_chunk(rowp, type, c * 8, false);
    }
    uint8_t* dst_row = tile + r * 128;
#pragma unroll
    for (int c = 0; c < HD / 8; c++)
        *reinterpret_cast<uint4*>(dst_row + (c >> 3) * kPanelBytes + (((c & 7) ^ (r & 7)) << 4)) = v[c];
}

// Coalesced forms of the two per-row transfers of a CTA.  A thread that moves its own row makes every warp instruction
// touch 32 rows (32 sectors for 16 bytes each); here a warp instruction covers whole rows, the row pointers travel by
// shuffle from the lanes that own them (lane i of warp w owns row 32w + i).
//
// F32 query rows -> f16 operand tile: per instruction RPI = 128 / HD rows, lane l reads float4 number l % (HD/4) of row
// l / (HD/4), converts and writes 8 bytes into the swizzled tile.  A null row pointer gives a zero row.
template <int HD>
__device__ __forceinline__ void load_q_rows_f32_coalesced(uint8_t* tile, int warp, int lane, const uint8_t* my_rowp) {
    constexpr int F4 = HD / 4, RPI = 32 / F4;   // float4 per row; rows per warp instruction
    const uint32_t plo = (uint32_t)reinterpret_cast<uintptr_t>(my_rowp), phi = (uint32_t)(reinterpret_cast<uintptr_t>(my_rowp) >> 32);
    const int c = lane % F4, sub = lane / F4;
#pragma unroll
    for (int batch = 0; batch < 32 / RPI / 16; batch++) {
        float4 f[16];
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const int src = (batch * 16 + k) * RPI + sub;
            const uintptr_t p = (uintptr_t)__shfl_sync(0xffffffffu, plo, src) | ((uintptr_t)__shfl_sync(0xffffffffu, phi, src) << 32);
            f[k] = p ? load_global(reinterpret_cast<const float4*>(p) + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const int row = warp * 32 + (batch * 16 + k) * RPI + sub;
            const int cc = c >> 1;   // 16-byte chunk of the f16 row
            *reinterpret_cast<uint2*>(tile + (cc >> 3) * kPanelBytes + row * 128 + (((cc & 7) ^ (row & 7)) << 4) + (c & 1) * 8) =
                make_uint2(pack_half2(f[k].x, f[k].y), pack_half2(f[k].z, f[k].w));
        }
    }
}

// The same for F16 query rows: a row is HD / 8 16-byte chunks, 256 / HD rows per warp instruction, copied as they are.
template <int HD>
__device__ __forceinline__ void load_q_rows_f16_coalesced(uint8_t* tile, int warp, int lane, const uint8_t* my_rowp) {
    constexpr int C16 = HD / 8, RPI = 32 / C16;
    const uint32_t plo = (uint32_t)reinterpret_cast<uintptr_t>(my_rowp), phi = (uint32_t)(reinterpret_cast<uintptr_t>(my_rowp) >> 32);
    const int cc = lane % C16, sub = lane / C16;
    uint4 v[32 / RPI];
#pragma unroll
    for (int k = 0; k < 32 / RPI; k++) {
        const int src = k * RPI + sub;
        const uintptr_t p = (uintptr_t)__shfl_sync(0xffffffffu, plo, src) | ((uintptr_t)__shfl_sync(0xffffffffu, phi, src) << 32);
        v[k] = p ? load_global(reinterpret_cast<const uint4*>(p) + cc) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int k = 0; k < 32 / RPI; k++) {
        const int row = warp * 32 + k * RPI + sub;
        *reinterpret_cast<uint4*>(tile + (cc >> 3) * kPanelBytes + row * 128 + (((cc & 7) ^ (row & 7)) << 4)) = v[k];
    }
}

// Output rows: each thread parks its scaled row in its warp's staging area (chunks swizzled by the row), then the warp
// writes whole rows.  `stage` is this warp's 32 * HD floats; a null row pointer skips the row.
template <int HD>
__device__ __forceinline__ void store_o_rows_coalesced(float* stage, int lane, float* my_out) {
    constexpr int F4 = HD / 4, RPI = 32 / F4;
    __syncwarp();
    const uint32_t plo = (uint32_t)reinterpret_cast<uintptr_t>(my_out), phi = (uint32_t)(reinterpret_cast<uintptr_t>(my_out) >> 32);
    const int c = lane % F4, sub = lane / F4;
#pragma unroll 4
    for (int k = 0; k < 32 / RPI; k++) {
        const int row = k * RPI + sub;
        const uintptr_t p = (uintptr_t)__shfl_sync(0xffffffffu, plo, row) | ((uintptr_t)__shfl_sync(0xffffffffu, phi, row) << 32);
        const float4 v = *reinterpret_cast<const float4*>(stage + row * HD + ((c ^ (row & 7)) << 2));
        if (p) *(reinterpret_cast<float4*>(p) + c) = v;
    }
}

// ---- parts that the two-CTA kernels share (fattn_tc5_h128.cuh) ------------------------------------------
// A query tile of F32 rows as tensor copies bring it: four panels of 128-byte swizzled rows, 32 columns each.  Columns 0 to 63 lie in the V stage
// and 64 to 127 in the operand tile itself: a softmax thread holds its whole row in registers before any of them writes the operand
// tile, and the first K tile is on its way meanwhile.
__device__ __forceinline__ constexpr int raw_panel_off(int p) { return (p < 2 ? 4 * kPanelBytes : 0) + (p & 1) * kPanelBytes; }

// Raw F32 row r -> F16 row r of the operand tile: 32 loads, 64 conversions, 16 stores per thread, all from shared memory.
__device__ __forceinline__ void convert_raw_row(uint8_t* smem_gen, int r) {
    uint4 row[16];
#pragma unroll
    for (int c = 0; c < 16; c++) {   // F16 chunk c = columns 8c .. 8c+7 = F32 chunks 2c, 2c+1 of raw panel c / 4
        const int f0 = (2 * c) & 7;
        const uint8_t* raw = smem_gen + raw_panel_off(c >> 2) + r * 128;
        const float4 x0 = *reinterpret_cast<const float4*>(raw + ((f0 ^ (r & 7)) << 4));
        const float4 x1 = *reinterpret_cast<const float4*>(raw + (((f0 + 1) ^ (r & 7)) << 4));
        row[c] = make_uint4(pack_half2(x0.x, x0.y), pack_half2(x0.z, x0.w), pack_half2(x1.x, x1.y), pack_half2(x1.z, x1.w));
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");   // the operand tile is written over raw columns 64 to 127 of all rows
#pragma unroll
    for (int c = 0; c < 16; c++) *reinterpret_cast<uint4*>(smem_gen + r * 128 + (c >> 3) * kPanelBytes + (((c & 7) ^ (r & 7)) << 4)) = row[c];
}

// S = Q.K^T of one key tile and O (+)= P.V, by one lane.
template <int HD>
__device__ __forceinline__ void issue_scores(uint32_t tmem_S, uint32_t q_lo, uint32_t k_lo) {
#pragma unroll
    for (int ks = 0; ks < HD / 16; ks++) {
        const uint32_t off16 = (uint32_t)(((ks >> 2) * kPanelBytes + (ks & 3) * 32) >> 4);
        mma_ss(tmem_S, desc64(q_lo + off16, smem_desc_hi(1024)), desc64(k_lo + off16, smem_desc_hi(1024)), idesc_f16(kTile, false), ks > 0 ? 1u : 0u);
    }
}
template <int HD>
__device__ __forceinline__ void issue_pv(uint32_t tmem_O, uint32_t tmem_P, uint32_t v_lo, bool first) {
    mma_ts(tmem_O, tmem_P, desc64(v_lo, smem_desc_hi(1024)), idesc_f16(HD, true), first ? 0u : 1u);
#pragma unroll
    for (int ks = 1; ks < kTile / 16; ks++) mma_ts(tmem_O, tmem_P + ks * 8, desc64(v_lo + ks * (2048 >> 4), smem_desc_hi(1024)), idesc_f16(HD, true), 1u);
}

// A first reference maximum of a row without a mask: that of its first 32 scores.  It is rarely more than 2^8 below the row's real maximum, and
// when it is (or when those columns are dead) the check behind softmax_tile has the tile redone against the exact maximum.
__device__ __forceinline__ float first_maximum(uint32_t s_row, int n_valid) {
    uint32_t s0[32];
    tmem_ld32(s_row, s0);
    tmem_wait_ld();
    float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        const float x0 = (i < n_valid) ? __uint_as_float(s0[i]) : -INFINITY;
        const float x1 = (i + 1 < n_valid) ? __uint_as_float(s0[i + 1]) : -INFINITY;
        m4[(i >> 1) & 3] = max3(m4[(i >> 1) & 3], x0, x1);
    }
    return max3(fmaxf(m4[0], m4[1]), m4[2], m4[3]);
}

// P = exp2(S * c - m) of a row's 128 scores, rounded to f16x2, their sum and the maximum of S, in one pass; columns >= n_valid are dead.  Rolling
// 32-column chunks: the load of chunk k+2 is issued into the registers chunk k has just left and completes under the exponentials of
// chunk k+1.  `meanwhile` runs behind the first chunk.
template <typename F>
__device__ __forceinline__ void softmax_tile(uint32_t s_row, float c, float m, bool full_tile, int n_valid, uint32_t (&preg)[2][32], float& mx, float& lsum, F meanwhile) {
    float mx8[8];
    uint64_t ls4[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
    for (int i = 0; i < 8; i++) mx8[i] = -INFINITY;
    const uint64_t c2 = pack2(c, c), nm2 = pack2(-m, -m);
    uint32_t sA[32], sB[32];
    // a partial tile (the last one, or the diagonal of a causal call) puts -inf into the dead columns first and skips chunks that are
    // dead for the whole warp: one copy of the arithmetic serves both
    auto chunk = [&](uint32_t (&sx)[32], uint32_t* p16, int col0) {
        if (!full_tile) {
            if (__all_sync(0xffffffffu, col0 >= n_valid)) {
#pragma unroll
                for (int i = 0; i < 16; i++) p16[i] = 0u;
                return;
            }
#pragma unroll
            for (int i = 0; i < 32; i++)
                if (col0 + i >= n_valid) sx[i] = 0xFF800000u;
        }
        softmax32(sx, p16, c2, nm2, mx8, ls4);
    };
    tmem_ld32(s_row, sA);
    tmem_ld32(s_row + 32, sB);
    tmem_wait_ld();
    chunk(sA, preg[0], 0);
    tmem_ld32(s_row + 64, sA);
    meanwhile();
    chunk(sB, preg[0] + 16, 32);
    tmem_wait_ld();
    tmem_ld32(s_row + 96, sB);
    chunk(sA, preg[1], 64);
    tmem_wait_ld();
    chunk(sB, preg[1] + 16, 96);
    mx = fmaxf(max3(fmaxf(mx8[0], mx8[1]), mx8[2], mx8[3]), max3(fmaxf(mx8[4], mx8[5]), mx8[6], mx8[7]));
    float l0, l1;
    unpack2(add2(add2(ls4[0], ls4[1]), add2(ls4[2], ls4[3])), l0, l1);
    lsum = l0 + l1;
}

template <int HD>
__device__ __forceinline__ void rescale_o(uint32_t o_row, float alpha) {
#pragma unroll
    for (int q4 = 0; q4 < HD / 32; q4++) {
        uint32_t oreg[32];
        tmem_ld32(o_row + q4 * 32, oreg);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; i++) oreg[i] = __float_as_uint(__uint_as_float(oreg[i]) * alpha);
        tmem_st32(o_row + q4 * 32, oreg);
    }
}

// A warp's 32 packed rows x 32 columns of the output are a box [32 columns, gqa heads, 32 / gqa tokens] of dst [hd, H, Tq, B]; the warp parks them
// as 128-byte rows with the 16-byte chunks swizzled by the row (the copy's own pattern, conflict-free for the stores) and one lane
// hands each panel to a tensor store, which also clips the tokens beyond Tq.  `stage`: this warp's 32 * HD floats; dead rows are written
// as literal zeros (whatever the padding row of Q held never reaches dst); `row0`: first packed row of the warp.
template <int HD>
__device__ __forceinline__ void store_o_box(const CUtensorMap& tmO, float* stage, uint32_t o_row, float inv, bool row_live, int lane, int row0, int rows_total, int hk,
                                            int gqa, int b) {
#pragma unroll
    for (int q4 = 0; q4 < HD / 32; q4++) {
        uint32_t oreg[32];
        tmem_ld32(o_row + q4 * 32, oreg);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<float4*>(stage + q4 * 32 * 32 + lane * 32 + (((i >> 2) ^ (lane & 7)) << 2)) =
                row_live ? make_float4(__uint_as_float(oreg[i]) * inv, __uint_as_float(oreg[i + 1]) * inv,
                                       __uint_as_float(oreg[i + 2]) * inv, __uint_as_float(oreg[i + 3]) * inv)
                         : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0 && row0 < rows_total) {
#pragma unroll
        for (int q4 = 0; q4 < HD / 32; q4++) tma_store_4d(&tmO, smem_u32(stage + q4 * 32 * 32), q4 * 32, hk * gqa, row0 / gqa, b);
        tma_store_commit_and_wait_read();
    }
}

// QMODE / OTMA: how the query tile comes in and the output tile goes out (see q_tma below).  Template parameters, not
// run-time flags: every path compiled into one kernel costs the others (the raw F32 form behind a flag took 5 % off the
// F16-Q encoder launches and 9 % off the T = 407 prefill).
template <int HD, int NSTG, bool HASMASK, int QMODE = 0, bool OTMA = false>
__global__ void __launch_bounds__(kThreadsTc5, 2)
fattn_prefill_tc5_kernel(const FattnArgs a, const __grid_constant__ CUtensorMap tmK,
                         const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmQ,
                         const __grid_constant__ CUtensorMap tmO) {
    constexpr int q_tma = QMODE;
    constexpr bool o_tma = OTMA;
    constexpr int PANELS = HD / 64;
    constexpr int TILE_BYTES = kPanelBytes * PANELS;

    extern __shared__ uint8_t smem_dyn[];
    const uint32_t smem_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_dyn + (smem_base - smem_u32(smem_dyn));
    const uint32_t sQ = smem_base;
    const uint32_t sK = sQ + TILE_BYTES;
    const uint32_t sV = sK + NSTG * TILE_BYTES;
    const uint32_t sBar = sV + NSTG * TILE_BYTES;  // 8-byte slots
    const uint32_t bar_k_full = sBar, bar_k_empty = sBar + 8 * NSTG, bar_v_full = sBar + 16 * NSTG,
                   bar_v_empty = sBar + 24 * NSTG, bar_s_full = sBar + 32 * NSTG, bar_p_ready = bar_s_full + 8,
                   bar_o_done = bar_s_full + 16, bar_pv_done = bar_s_full + 24, bar_q_full = bar_s_full + 32, bar_q_conv = bar_s_full + 40;
    uint8_t* misc = smem_gen + (1 + 2 * NSTG) * TILE_BYTES + 32 * NSTG + 64;
    // q_tma: 0 = the softmax warps load and convert the Q tile; 1 = F16 rows by one tensor copy into the operand tile;
    // 2 = F32 rows by tensor copies into stages that are not needed yet, converted from there by the softmax warps.
    constexpr bool q_raw = QMODE == 2;
    static_assert(!q_raw || (HD == 128 && NSTG == 1), "the raw tile takes the stages of head_dim 128");
    // head_dim 64 leaves 64 spare TMEM columns: P gets its own, so S of the next tile can be issued before P.V
    constexpr bool SEP_P = (HD == 64);
    volatile uint32_t* s_tmem_base = reinterpret_cast<volatile uint32_t*>(misc);
    volatile int* s_abort = reinterpret_cast<volatile int*>(misc + 4);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // Causal launches hand out the query tiles with the most KV tiles first (longest-processing-time order over
    // the whole grid: the tile index becomes the slowest-varying coordinate, reversed), which shortens the tail of
    // short prefills; otherwise consecutive CTAs are the query tiles of one head, which share K/V in L2.
    // GQA packing: the grid runs over KV heads, and a CTA's 128 rows are (query position, head of the group) pairs -
    // packed row q0 + r is query (q0 + r) / gqa of head hk*gqa + (q0 + r) % gqa.  The heads of a group share their
    // K/V tiles, and a short causal prefill covers fewer, fuller tiles (gqa = 1: the plain one-head tile).
    int q0 = blockIdx.x * kTile, hk = blockIdx.y, b = blockIdx.z;
    if (a.causal) {
        const int lin = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z), hb = gridDim.y * gridDim.z;
        q0 = (gridDim.x - 1 - lin / hb) * kTile;
        hk = (lin % hb) % gridDim.y, b = (lin % hb) / gridDim.y;
    }
    // While the previous kernel runs (behind a conversion of K and V, say, which lets this one become resident early) the query tile is
    // brought into L2, from where its copy behind the wait is half as far: 8 streams x 407 tokens over a Q8_0 cache, F32
    // queries, 53.6 -> 51.9 us per layer; 16 x 100 tokens 18.1 -> 17.5.  Behind any other kernel, and in CTAs of later waves, it runs
    // ahead of the TMEM allocation and the barriers: F32 queries gain 2 % (16 x 407 tokens over F16 rows 75.0 -> 73.8, 1 x 407 14.3 ->
    // 14.0), F16 queries as much as they lose (1 x 407 12.4 -> 12.35, 16 x 407 60.7 -> 60.5, masked rows of head_dim 64, 1 x 224, 12.9
    // -> 12.75; but 16 x 100 16.8 -> 17.0, 16 x 750 not causal 102.4 -> 103.3, where leaving out the CTAs of later waves gave half
    // of that back and took the other gains).  (The tile of the CTA that follows on this SM, asked for as well, cost the gain again:
    // it competes with the copies that are waited for.)
    if (QMODE && tid == 4 * 32) {
        constexpr int kCols = QMODE == 2 ? 32 : 64;
#pragma unroll
        for (int p = 0; p < HD / kCols; p++) tma_prefetch_4d(&tmQ, p * kCols, hk * a.gqa, q0 / a.gqa, b);
    }
    // launched with programmatic stream serialisation: nothing is read or written before the previous kernel of the
    // stream has completed and flushed
    const uint32_t behind_wait = wait_for_predecessors();
    const int bk = b / a.bq;
    const int rows_total = a.Tq * a.gqa;   // packed rows of this (kv head, batch entry)
    const int tq_b = q_rows_of(a, b);      // query rows at or beyond it are padding of a batched launch: zeros
    const int rows_live = tq_b * a.gqa;

    int len_b = a.Lk;
    if (a.kv_len) {
        const int v = a.kv_len[b];
        len_b = v < 0 ? 0 : (v > a.Lk ? a.Lk : v);
    }
    const int n_past = n_past_of(a, len_b, tq_b);
    int kmax = q0 < rows_live ? len_b : 0;   // a tile of padding rows reads no keys
    if (a.causal) kmax = min(kmax, n_past + min((q0 + kTile - 1) / a.gqa + 1, tq_b));
    const int n_tiles = kmax > 0 ? (kmax + kTile - 1) / kTile : 0;

    if (n_tiles == 0) {  // nothing to attend to: zeros
        if (tid < kTile && q0 + tid < rows_total) {
            const int iq = (q0 + tid) / a.gqa, h = hk * a.gqa + (q0 + tid) % a.gqa;
            float4* out = reinterpret_cast<float4*>(a.dst + (((int64_t)b * a.Tq + iq) * a.dst_heads + h) * HD);
#pragma unroll
            for (int i = 0; i < HD / 4; i++) out[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        return;
    }

    // ---- set-up ----
    if (tid == 4 * 32) {
        for (int i = 0; i < NSTG; i++) {
            mbar_init(bar_k_full + 8 * i, 1);
            mbar_init(bar_k_empty + 8 * i, 1);
            mbar_init(bar_v_full + 8 * i, 1);
            mbar_init(bar_v_empty + 8 * i, 1);
        }
        mbar_init(bar_s_full, 1);
        mbar_init(bar_p_ready, 4);   // one arrival per softmax warp
        mbar_init(bar_o_done, 1);
        mbar_init(bar_pv_done, 1);
        mbar_init(bar_q_full, 1);
        mbar_init(bar_q_conv, 4);    // one arrival per softmax warp
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (q_raw) {
            // HD / 32 panels of 128 rows x 32 floats, rows in packed order like the F16 box
            mbar_arrive_expect_tx(bar_q_full, (HD / 32) * kPanelBytes);
#pragma unroll
            for (int p = 0; p < HD / 32; p++)
                tma_load_4d(sQ + raw_panel_off(p), &tmQ, bar_q_full, p * 32, hk * a.gqa, q0 / a.gqa, b);
        } else if (q_tma) {
            // F16 query rows go straight into the operand layout: one copy instead of a pass through the softmax warps'
            // registers, which a CTA sharing its SM with another one in its key loop executes at a few tens of clocks
            // per instruction.  The box is [64 columns, the gqa heads of the group, 128 / gqa tokens]: its rows land in
            // packed order (token-major, head of the group minor).  Tokens at or beyond Tq read as zeros.
            mbar_arrive_expect_tx(bar_q_full, TILE_BYTES);
#pragma unroll
            for (int p = 0; p < PANELS; p++) tma_load_4d(sQ + p * kPanelBytes, &tmQ, bar_q_full, p * 64, hk * a.gqa, q0 / a.gqa, b);
        }
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmK)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmV)) : "memory");
        // the first NSTG tiles need no empty-slot wait: start their copies before the CTA-wide set-up barrier
        for (int j = 0; j < NSTG && j < n_tiles; j++) {
            mbar_arrive_expect_tx(bar_k_full + 8 * j, TILE_BYTES);
#pragma unroll
            for (int p = 0; p < PANELS; p++)
                tma_load_4d(sK + j * TILE_BYTES + p * kPanelBytes, &tmK, bar_k_full + 8 * j, p * 64, j * kTile, hk, bk);
            if (q_raw) continue;   // the V stage holds raw Q rows for now
            mbar_arrive_expect_tx(bar_v_full + 8 * j, TILE_BYTES);
#pragma unroll
            for (int p = 0; p < PANELS; p++)
                tma_load_4d(sV + j * TILE_BYTES + p * kPanelBytes, &tmV, bar_v_full + 8 * j, p * 64, j * kTile, hk, bk);
        }
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(const_cast<uint32_t*>(s_tmem_base))),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (warp < 4 && !q_tma) {
        // Q tile -> shared memory (thread r writes row r)
        const int r = tid;
        const int iq = (q0 + r) / a.gqa, h = hk * a.gqa + (q0 + r) % a.gqa;
        const uint8_t* rowp = a.q.p + (int64_t)iq * a.q.nb1 + (int64_t)h * a.q.nb2 + (int64_t)b * a.q.nb3;
        if (a.q.type == B200_TYPE_F32 && a.q.vec16) load_q_rows_f32_coalesced<HD>(smem_gen, warp, lane, q0 + r < rows_total ? rowp : nullptr);
        else if (a.q.type == B200_TYPE_F16 && a.q.vec16) load_q_rows_f16_coalesced<HD>(smem_gen, warp, lane, q0 + r < rows_total ? rowp : nullptr);
        else load_q_row<HD>(smem_gen, r, rowp, a.q.type, a.q.vec16 != 0, q0 + r < rows_total);
        fence_proxy_async();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *s_tmem_base, 0);
    const uint32_t tmem_S = tmem_base;            // cols [0,128)
    const uint32_t tmem_P = SEP_P ? tmem_base + kTile + HD : tmem_base;  // f16x2: cols [192,256) (hd 64) or aliasing S [0,64)
    const uint32_t tmem_O = tmem_base + kTile;    // cols [128,128+HD)
    if constexpr (q_raw) {
        if (q_raw && warp < 4) {
            const bool there = mbar_wait(bar_q_full, 0, s_abort);
            convert_raw_row(smem_gen, tid);
            if (there) {
                fence_proxy_async();   // the operand tile is read, and the V stage is overwritten, through the async proxy
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_q_conv);
            }
        }
    }

    if (warp == 4) {
        // ================= TMA producer =================
        if (lane == 0) {
            bool ok = true;
            int issued_k = min(NSTG, n_tiles), issued_v = q_raw ? 0 : min(NSTG, n_tiles);
            if (q_raw) {
                ok = mbar_wait(bar_q_conv, 0, s_abort);
                for (int j = 0; j < NSTG && j < n_tiles && ok; j++) {
                    mbar_arrive_expect_tx(bar_v_full + 8 * j, TILE_BYTES);
#pragma unroll
                    for (int p = 0; p < PANELS; p++)
                        tma_load_4d(sV + j * TILE_BYTES + p * kPanelBytes, &tmV, bar_v_full + 8 * j, p * 64, j * kTile, hk, bk);
                    issued_v = j + 1;
                }
            }
            for (int j = NSTG; j < n_tiles && ok; j++) {
                const int slot = j % NSTG, use = j / NSTG;
                const int k0 = j * kTile;
                ok = mbar_wait(bar_k_empty + 8 * slot, (use - 1) & 1, s_abort);
                if (!ok) break;
                mbar_arrive_expect_tx(bar_k_full + 8 * slot, TILE_BYTES);
#pragma unroll
                for (int p = 0; p < PANELS; p++)
                    tma_load_4d(sK + slot * TILE_BYTES + p * kPanelBytes, &tmK, bar_k_full + 8 * slot, p * 64, k0, hk, bk);
                issued_k = j + 1;
                ok = mbar_wait(bar_v_empty + 8 * slot, (use - 1) & 1, s_abort);
                if (!ok) break;
                mbar_arrive_expect_tx(bar_v_full + 8 * slot, TILE_BYTES);
#pragma unroll
                for (int p = 0; p < PANELS; p++)
                    tma_load_4d(sV + slot * TILE_BYTES + p * kPanelBytes, &tmV, bar_v_full + 8 * slot, p * 64, k0, hk, bk);
                issued_v = j + 1;
            }
            if (!ok) {
                // drain: wait (bounded) for the copies this thread still has in flight
                if (q_tma)
                    for (uint32_t it = 0; it < 4096 && !mbar_try_wait(bar_q_full, 0); ++it) __nanosleep(256);
                for (int j = max(0, issued_k - NSTG); j < issued_k; j++)
                    for (uint32_t it = 0; it < 4096 && !mbar_try_wait(bar_k_full + 8 * (j % NSTG), (j / NSTG) & 1); ++it) __nanosleep(256);
                for (int j = max(0, issued_v - NSTG); j < issued_v; j++)
                    for (uint32_t it = 0; it < 4096 && !mbar_try_wait(bar_v_full + 8 * (j % NSTG), (j / NSTG) & 1); ++it) __nanosleep(256);
            }
        }
    } else if (warp == 5) {
        // ================= MMA issuer =================
        // Order: S[0]; then per tile j: (barriers of tile j+1 are awaited while the softmax of tile j runs)
        // wait P[j] -> PV[j] -> S[j+1], back to back, so the softmax threads of the next tile wake as early
        // as the tensor pipe allows.  S[j+1] overwrites the columns P[j] lives in; tcgen05.mma executes in
        // issue order, so PV[j] has consumed P[j] before S[j+1] writes.
        {
            const uint32_t q_lo = smem_desc_lo(sQ, 16), k_lo = smem_desc_lo(sK, 16), v_lo = smem_desc_lo(sV, kPanelBytes);
            auto issue_s = [&](int slot) {
                issue_scores<HD>(tmem_S, q_lo, k_lo + slot * (TILE_BYTES >> 4));
                tc_commit(bar_s_full);
            };
            bool ok = mbar_wait(bar_k_full, 0, s_abort);
            if (ok && q_tma) ok = mbar_wait(q_raw ? bar_q_conv : bar_q_full, 0, s_abort);
            ok = warp_all(ok);
            if (ok) {
                tc_fence_after();
                if (elect_one()) {
                    issue_s(0);
                    tc_commit(bar_k_empty);
                }
                __syncwarp();
            }
            for (int j = 0; j < n_tiles && ok; j++) {
                const int slot = j % NSTG, use = j / NSTG;
                const int nslot = (j + 1) % NSTG, nuse = (j + 1) / NSTG;
                const bool more = j + 1 < n_tiles;
                ok = mbar_wait(bar_v_full + 8 * slot, use & 1, s_abort);
                if (ok && more) ok = mbar_wait(bar_k_full + 8 * nslot, nuse & 1, s_abort);
                if (ok) ok = mbar_wait(bar_p_ready, j & 1, s_abort);
                ok = warp_all(ok);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    // with P in its own columns the next S goes first: the softmax threads wake after 4 MMAs, not 12
                    if (SEP_P && more) issue_s(nslot);
                    issue_pv<HD>(tmem_O, tmem_P, v_lo + slot * (TILE_BYTES >> 4), j == 0);
                    if (SEP_P) {
                        if (more) tc_commit(bar_k_empty + 8 * nslot);   // after the P.V MMAs: off the softmax threads' critical path
                        tc_commit(bar_v_empty + 8 * slot);
                        tc_commit(bar_pv_done);
                    } else {
                        tc_commit(bar_v_empty + 8 * slot);
                        if (more) {
                            issue_s(nslot);
                            tc_commit(bar_k_empty + 8 * nslot);
                        }
                    }
                    if (!more) tc_commit(bar_o_done);
                }
                __syncwarp();
            }
            if (!ok) {
                // make sure no MMA of this CTA is still running before TMEM is released (the commit comes from the lane that
                // issued them)
                if (elect_one()) tc_commit(bar_o_done);
                __syncwarp();
                for (uint32_t it = 0; it < 65536 && !mbar_try_wait(bar_o_done, 0); ++it) __nanosleep(256);
            }
            __syncwarp();
        }
    } else {
        // ================= softmax / correction / epilogue =================
        const int r = tid;
        const bool row_live = q0 + r < rows_live;
        const bool row_zero = !row_live && q0 + r < rows_total;   // a padding row inside the tensor: its dst row is zero-filled
        const int iq_dst = (q0 + r) / a.gqa;
        const int iq = row_live ? iq_dst : a.Tq, h = hk * a.gqa + (q0 + r) % a.gqa;   // dead rows: iq = Tq
        const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
        const float c = a.scale * kLog2e;
        int kend = len_b;
        if (a.causal) kend = min(kend, n_past + iq + 1);
        float m_ref = -INFINITY, l_run = 0.0f;
        bool ok = true;
        // explicit mask row of this query ([Lk, Tq, 1|H, 1|B] F16); rows past Tq reuse row 0
        const uint8_t* mrow = HASMASK ? a.mask.p + behind_wait + (int64_t)(iq < a.Tq ? iq : 0) * a.mask.nb1 +
                                            (int64_t)(h % a.mask_ne2) * a.mask.nb2 + (int64_t)(b % a.mask_ne3) * a.mask.nb3
                                      : nullptr;
        const float c_exp = HASMASK ? 1.0f : c;   // with a mask the scores are moved to the log2 domain by apply_mask64
        for (int j = 0; j < n_tiles; j++) {
            ok = mbar_wait(bar_s_full, j & 1, s_abort);
            if (!ok) break;
            tc_fence_after();
            const int n_valid = kend - j * kTile;  // columns >= n_valid of this row are masked
            const bool full_tile = __all_sync(0xffffffffu, n_valid >= kTile);
            if (j == 0) {
                // First tile: a first reference maximum
                float mx = -INFINITY;
                if (HASMASK) {
#pragma unroll
                    for (int hh = 0; hh < 2; hh++) {
                        uint32_t sreg[2][32];
                        tmem_ld32(tmem_S + lane_base + hh * 64, sreg[0]);
                        tmem_ld32(tmem_S + lane_base + hh * 64 + 32, sreg[1]);
                        tmem_wait_ld();
                        apply_mask64(sreg, mrow + (int64_t)(j * kTile + hh * 64) * 2, a.Lk - (j * kTile + hh * 64), c);
                        mx = fmaxf(mx, row_max64(sreg, hh * 64, full_tile ? 2 * kTile : n_valid));
                    }
                } else {
                    mx = first_maximum(tmem_S + lane_base, n_valid);
                }
                m_ref = mx * c_exp;  // c > 0
            }
            uint32_t preg[2][32];
            float lsum = 0.0f;
            bool pv_waited = false;
            uint32_t pv_probe = 0;   // early answer to "has P.V of the previous tile completed" (it normally has by mid-tile)
            for (int attempt = 0; attempt < 2; attempt++) {
                // P = exp2(S*c - m_ref), rounded to f16x2; the tile maximum is tracked in the same pass and
                // only checked afterwards (lazy rescale).
                const float m_use = (m_ref == -INFINITY) ? 0.0f : m_ref;
                float mx = -INFINITY;
                lsum = 0.0f;
                if constexpr (!HASMASK) {
                    softmax_tile(tmem_S + lane_base, c_exp, m_use, full_tile, n_valid, preg, mx, lsum, [&]() {
                        if (SEP_P && j > 0 && !pv_waited && !pv_probe) pv_probe = mbar_test(bar_pv_done, (j - 1) & 1);
                    });
                } else
#pragma unroll
                for (int hh = 0; hh < 2; hh++) {
                    uint32_t sreg[2][32];
                    tmem_ld32(tmem_S + lane_base + hh * 64, sreg[0]);
                    tmem_ld32(tmem_S + lane_base + hh * 64 + 32, sreg[1]);
                    if (SEP_P && hh == 1 && j > 0 && !pv_waited && !pv_probe) pv_probe = mbar_test(bar_pv_done, (j - 1) & 1);
                    tmem_wait_ld();
                    uint4 mv[8];
                    load_mask64(mv, mrow + (int64_t)(j * kTile + hh * 64) * 2, a.Lk - (j * kTile + hh * 64));
                    if (full_tile) softmax64_masked<false>(sreg, mv, preg[hh], c, m_use, 0, 0, mx, lsum);
                    else softmax64_masked<true>(sreg, mv, preg[hh], c, m_use, hh * 64, n_valid, mx, lsum);
                }
                const float m_tile = HASMASK ? mx + m_use : mx * c_exp;   // (the masked form tracks the maximum of x = logit - m)
                const bool grow = m_tile > m_ref + kRescaleThreshold;
                if (!__any_sync(0xffffffffu, grow)) break;
                // some row of this warp outgrew its reference maximum: rescale O and l, then redo P
                if (SEP_P && j > 0 && !pv_waited) {  // O must be at rest: P.V of the previous tile has completed
                    ok = mbar_wait(bar_pv_done, (j - 1) & 1, s_abort);
                    if (!ok) break;
                    tc_fence_after();
                    pv_waited = true;
                }
                const float m_new = fmaxf(m_ref, m_tile);
                const float alpha = (m_new == -INFINITY) ? 1.0f : ex2(m_ref - m_new);
                l_run *= alpha;
                if (j > 0) rescale_o<HD>(tmem_O + lane_base, alpha);
                m_ref = m_new;
            }
            if (!ok) break;
            l_run += lsum;
            if (SEP_P && j > 0 && !pv_waited) {  // P[j-1] must have been consumed before P[j] overwrites it
                if (!pv_probe) ok = mbar_wait(bar_pv_done, (j - 1) & 1, s_abort);
                if (!ok) break;
                tc_fence_after();
            }
            tmem_st32(tmem_P + lane_base, preg[0]);
            tmem_st32(tmem_P + lane_base + 32, preg[1]);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_p_ready);
        }
        if (ok) ok = mbar_wait(bar_o_done, 0, s_abort);
        if (ok) {
            tc_fence_after();
            // dead rows are written as literal zeros, rows outside the tensor not at all.  The K/V stages are free once the last MMA has
            // completed: they stage O.
            const float inv = row_live && l_run > 0.0f ? 1.0f / l_run : 0.0f;
            float* out = (row_live || row_zero) ? a.dst + (((int64_t)b * a.Tq + iq_dst) * a.dst_heads + h) * HD : nullptr;
            float* stage = reinterpret_cast<float*>(smem_gen + TILE_BYTES) + warp * 32 * HD;
            if (o_tma) {
                store_o_box<HD>(tmO, stage, tmem_O + lane_base, inv, row_live, lane, q0 + warp * 32, rows_total, hk, a.gqa, b);
            } else {
#pragma unroll
                for (int q4 = 0; q4 < HD / 32; q4++) {
                    uint32_t oreg[32];
                    tmem_ld32(tmem_O + lane_base + q4 * 32, oreg);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        *reinterpret_cast<float4*>(stage + lane * HD + ((((q4 * 32 + i) >> 2) ^ (lane & 7)) << 2)) =
                            row_live ? make_float4(__uint_as_float(oreg[i]) * inv, __uint_as_float(oreg[i + 1]) * inv,
                                                   __uint_as_float(oreg[i + 2]) * inv, __uint_as_float(oreg[i + 3]) * inv)
                                     : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                store_o_rows_coalesced<HD>(stage, lane, out);
            }
        }
    }

    // ---- teardown ----
    tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

// ---- host side ----------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static std::once_flag once;
    static EncodeTiledFn fn = nullptr;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    });
    return fn;
}

// K/V as a rank-4 F16 tensor [hd, Lk, Hkv, Bk] with the caller's byte strides; box = 64 columns x `keys` rows x 1 x 1.
bool encode_kv_map(CUtensorMap* m, const View& v, int hd, int Lk, int Hkv, int Bk, int keys = kTile) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)hd, (cuuint64_t)Lk, (cuuint64_t)Hkv, (cuuint64_t)Bk};
    const cuuint64_t strides[3] = {(cuuint64_t)v.nb1, (cuuint64_t)v.nb2, (cuuint64_t)v.nb3};
    const cuuint32_t box[4] = {64, (cuuint32_t)keys, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<uint8_t*>(v.p), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Q as a rank-4 F16 or F32 tensor [hd, H, Tq, B] (head stride nb2, token stride nb1); box = 128 bytes of columns x the gqa
// heads of a group x 128 / gqa tokens: the rows of a box are the packed rows of a query tile.
bool encode_q_map(CUtensorMap* m, const FattnArgs& a) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)a.hd, (cuuint64_t)a.H, (cuuint64_t)a.Tq, (cuuint64_t)a.B};
    const cuuint64_t strides[3] = {(cuuint64_t)a.q.nb2, (cuuint64_t)a.q.nb1, (cuuint64_t)a.q.nb3};
    const bool f32 = a.q.type == B200_TYPE_F32;   // 128-byte box rows either way: 64 halves or 32 floats
    const cuuint32_t box[4] = {f32 ? 32u : 64u, (cuuint32_t)a.gqa, (cuuint32_t)(kTile / a.gqa), 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return fn(m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<uint8_t*>(a.q.p), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// dst as a rank-4 F32 tensor [hd, H, Tq, B] (contiguous); box = 32 columns x gqa heads x 32 / gqa tokens: a warp's
// 32 packed rows.
bool encode_o_map(CUtensorMap* m, const FattnArgs& a) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)a.hd, (cuuint64_t)a.H, (cuuint64_t)a.Tq, (cuuint64_t)a.B};
    const cuuint64_t strides[3] = {(cuuint64_t)a.hd * 4, (cuuint64_t)a.hd * 4 * a.dst_heads, (cuuint64_t)a.hd * 4 * a.dst_heads * a.Tq};
    const cuuint32_t box[4] = {32, (cuuint32_t)a.gqa, (cuuint32_t)(32 / a.gqa), 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a.dst, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// R as a rank-4 F16 tensor [hd, 2T-1, H, 1|B]; box = 64 columns x `rows` rows.
bool encode_r_map(CUtensorMap* m, const FattnArgs& a, int rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const int64_t nb3 = a.r_ne3 > 1 ? a.r.nb3 : a.r.nb2 * a.H;
    const cuuint64_t dims[4] = {(cuuint64_t)a.hd, (cuuint64_t)(2 * a.Tq - 1), (cuuint64_t)a.H, (cuuint64_t)a.r_ne3};
    const cuuint64_t strides[3] = {(cuuint64_t)a.r.nb1, (cuuint64_t)a.r.nb2, (cuuint64_t)nb3};
    const cuuint32_t box[4] = {64, (cuuint32_t)rows, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<uint8_t*>(a.r.p), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Launch that may begin while the previous kernel of the stream drains, if that kernel allows it
// (griddepcontrol.launch_dependents: the conversion pre-pass, the cache append and others do).  The kernels wait for the predecessor's
// completion (griddepcontrol.wait) before they read anything it may have written.
// `cluster` > 1: so many CTAs along x form a thread-block cluster.
template <typename Kern, typename... Args>
cudaError_t launch_pdl_cluster(Kern kern, dim3 grid, int cluster, int threads, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster, attr[1].val.clusterDim.y = 1, attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}
template <typename Kern, typename... Args>
cudaError_t launch_pdl(Kern kern, dim3 grid, int threads, size_t smem, cudaStream_t st, Args... args) {
    return launch_pdl_cluster(kern, grid, 1, threads, smem, st, args...);
}

#include "fattn_tc5_relpos.cuh"

int launch_relpos(const FattnArgs& a, cudaStream_t st, char* errbuf, size_t errlen) {
    CUtensorMap tmK, tmV, tmR;
    if (!encode_kv_map(&tmK, a.k, a.hd, a.Lk, a.Hkv, a.B / a.bq) || !encode_kv_map(&tmV, a.v, a.hd, a.Lk, a.Hkv, a.B / a.bq) ||
        !encode_r_map(&tmR, a, kRelBlock)) {
        snprintf(errbuf, errlen, "cuTensorMapEncodeTiled failed for K/V/R");
        return B200_E_CUDA;
    }
    cudaError_t e;
    dim3 grid((a.Tq + kTile - 1) / kTile, a.H, a.B);
    static bool set[2][64] = {};
    auto go = [&](auto kern, bool (&smem_set)[64]) {
        e = set_smem_once(kern, kRelSmem, smem_set);
        if (e == cudaSuccess) e = launch_pdl(kern, grid, kThreadsRelpos, kRelSmem, st, a, 1.0f / a.scale, tmK, tmV, tmR);
    };
    if (a.has_mask) go(fattn_prefill_tc5_relpos_kernel<true>, set[0]);
    else go(fattn_prefill_tc5_relpos_kernel<false>, set[1]);
    if (e != cudaSuccess) {
        snprintf(errbuf, errlen, "tcgen05 rel-pos prefill launch: %s", cudaGetErrorString(e));
        return B200_E_CUDA;
    }
    return B200_OK;
}

#include "fattn_tc5_h64.cuh"
#include "fattn_tc5_h128.cuh"

// One instantiation per kernel: its own "shared-memory attribute raised" flags per device.
template <auto Kern, typename... Args>
cudaError_t launch_inst(dim3 grid, size_t smem, cudaStream_t st, Args... args) {
    static bool smem_set[64] = {false};
    cudaError_t e = set_smem_once(Kern, smem, smem_set);
    if (e == cudaSuccess) e = launch_pdl(Kern, grid, kThreadsTc5, smem, st, args...);
    return e;
}

// Whether the query rows / the output rows of a launch can travel as boxes of [columns, heads of the group, tokens]: the
// rows of a warp (32 packed rows) are then whole tokens.
bool gqa_box(const FattnArgs& a) { return a.gqa >= 1 && a.gqa <= 32 && 32 % a.gqa == 0; }
bool q_box_ok(const FattnArgs& a) {
    return a.q.vec16 && gqa_box(a) && !a.bias_u && a.q.nb1 % 16 == 0 && a.q.nb2 % 16 == 0 && a.q.nb3 % 16 == 0 && a.q.nb1 > 0 && a.q.nb2 > 0 &&
           a.q.nb3 > 0;
}

// How a head_dim 64 launch without a mask runs, from its query tiles and its keys: n >= 1 CTAs (a cluster of 1, 2, 4 or 8)
// of the four-CTA kernel share a tile's 64-key steps, 0 = the two-CTA kernel with 128-key tiles.  A CTA's time is a start and its
// steps, both by how many CTAs its SM holds; sharing a tile costs 3.4 us more (two cluster barriers, O through shared
// memory, the merge).  Clusters do not fill every SM: 72 of two and 32 of four or eight CTAs run side by side before
// SMs take a second CTA.  The two-CTA kernel has the shorter chain per key when an SM holds one CTA.
// Fitted to 172 shapes (1 to 6 windows, 6 to 20 heads, 150 to 1500 frames; device time by CUDA graph): never more than 6 % above
// the best of the five.  In us, two-CTA kernel / one / two / four / eight CTAs per tile: 64 tiles of 16 steps 15.0 / 16.7 / 13.5 /
// 12.0 / 14.8; 96 of 24 20.3 / 23.2 / 19.4 / 16.6 / 21.7; 96 of 8 9.9 / 10.4 / 12.3 / 12.0 / 17.5; 144 of 24 20.8 / 23.4 / 19.9 /
// 24.0 / 28.9; 144 of 16 15.6 / 17.2 / 16.3 / 20.1 / 26.0; 192 of 24 25.6 / 26.2 / 24.2 / 27.8 / 35.9; 288 of 11 15.4 / 15.3 / 19.9 /
// 28.3 / 44.4.
int h64_plan(long tiles, int keys, bool causal) {
    constexpr double kStepUs[5] = {0.0, 0.83, 0.93, 1.2, 1.49}, kStartUs[5] = {0.0, 3.7, 4.8, 5.9, 6.6};
    const int steps = (keys + kH64Keys - 1) / kH64Keys, pairs = (keys + kTile - 1) / kTile;   // 64-key steps, 128-key tiles
    // A causal launch is as long as its last query tiles, which start first; up to two CTAs per SM (an eighth more when the
    // tiles that wait are short against the rest) the two-CTA kernel runs those faster: 160 tiles of 16 steps 15.3 / 18.0 us,
    // 240 of 24 21.4 / 24.3, 288 of 8 10.9 / 11.5, 320 of 16 17.9 / 18.9; but 240 of 5 9.2 / 9.2, 320 of 8 14.6 / 12.5.
    if (causal && tiles > 148 && tiles <= (pairs >= 8 ? 333 : 296) && pairs >= 4) return 0;
    if (tiles > 2 * 148) return 1;
    int best = 1;
    double best_cost = 0.0;
    for (int n = 1; n <= 8; n *= 2) {
        const long places = n == 1 ? 148 : (n == 2 ? 144 : 128), per_sm = (tiles * n + places - 1) / places;
        if (per_sm > 4) break;   // more than one wave
        const double cost = (steps + n - 1) / n * kStepUs[per_sm] + kStartUs[per_sm] + (n > 1 ? 3.4 : 0.0);
        // (a clear gain only: where it is even, the result of an entry stays what it is inside a larger batch, bit for bit)
        if (n == 1 || cost < 0.96 * best_cost) best = n, best_cost = cost;
    }
    const double two_cta = 4.5 + 1.32 * pairs;   // one CTA per SM; with two per SM it gains no more than 2 %
    return tiles <= 148 && two_cta < 0.98 * best_cost ? 0 : best;
}

int launch_h64(const FattnArgs& a, int n_split, cudaStream_t st, char* errbuf, size_t errlen) {
    CUtensorMap tmK, tmV;
    if (!encode_kv_map(&tmK, a.k, a.hd, a.Lk, a.Hkv, a.B / a.bq, kH64Keys) || !encode_kv_map(&tmV, a.v, a.hd, a.Lk, a.Hkv, a.B / a.bq, kH64Keys)) {
        snprintf(errbuf, errlen, "cuTensorMapEncodeTiled failed for K/V");
        return B200_E_CUDA;
    }
    CUtensorMap tmQ = tmK, tmO = tmK;
    const bool q_tma = a.q.type == B200_TYPE_F16 && q_box_ok(a) && encode_q_map(&tmQ, a);
    const bool o_tma = gqa_box(a) && !a.dst_on_host && (uintptr_t)a.dst % 16 == 0 && encode_o_map(&tmO, a);
    FattnArgs as = a;
    const int n_q = (a.Tq * a.gqa + kTile - 1) / kTile;
    as.n_splits = n_split;
    dim3 grid(n_q * as.n_splits, a.Hkv, a.B);
    auto go = [&](auto kern, bool (&smem_set)[64]) {
        cudaError_t e = set_smem_once(kern, kH64Smem, smem_set);
        if (e == cudaSuccess) e = launch_pdl_cluster(kern, grid, as.n_splits, kH64Threads, kH64Smem, st, as, tmK, tmV, tmQ, tmO);
        return e;
    };
    static bool set[6][64] = {};
    cudaError_t e;
    if (as.n_splits > 1) e = q_tma ? go(fattn_prefill_tc5_h64_kernel<true, false, true>, set[4]) : go(fattn_prefill_tc5_h64_kernel<false, false, true>, set[5]);
    else e = q_tma ? (o_tma ? go(fattn_prefill_tc5_h64_kernel<true, true>, set[0]) : go(fattn_prefill_tc5_h64_kernel<true, false>, set[1]))
                   : (o_tma ? go(fattn_prefill_tc5_h64_kernel<false, true>, set[2]) : go(fattn_prefill_tc5_h64_kernel<false, false>, set[3]));
    if (e != cudaSuccess) {
        snprintf(errbuf, errlen, "tcgen05 prefill launch: %s", cudaGetErrorString(e));
        return B200_E_CUDA;
    }
    return B200_OK;
}

template <int HD, int NSTG>
int launch_t(const FattnArgs& a_in, cudaStream_t st, char* errbuf, size_t errlen) {
    const FattnArgs& a = a_in;
    CUtensorMap tmK, tmV;
    if (!encode_kv_map(&tmK, a.k, a.hd, a.Lk, a.Hkv, a.B / a.bq) || !encode_kv_map(&tmV, a.v, a.hd, a.Lk, a.Hkv, a.B / a.bq)) {
        snprintf(errbuf, errlen, "cuTensorMapEncodeTiled failed for K/V");
        return B200_E_CUDA;
    }
    constexpr int TILE_BYTES = kPanelBytes * (HD / 64);
    const size_t smem = 1024 + (size_t)(1 + 2 * NSTG) * TILE_BYTES + 32 * NSTG + 64 + 8;
    constexpr bool RAW_INST = HD == 128 && NSTG == 1;   // the raw F32 form exists (and pays) at head_dim 128 only
    CUtensorMap tmQ = tmK;
    int q_tma = 0;
    if (a.q.type == B200_TYPE_F16 && q_box_ok(a)) q_tma = encode_q_map(&tmQ, a) ? 1 : 0;
    else if (RAW_INST && a.q.type == B200_TYPE_F32 && q_box_ok(a)) q_tma = encode_q_map(&tmQ, a) ? 2 : 0;   // F32 rows: raw tile into stages not needed yet, converted from shared memory
    CUtensorMap tmO = tmK;
    const bool o_tma = gqa_box(a) && !a.dst_on_host && (uintptr_t)a.dst % 16 == 0 && encode_o_map(&tmO, a);   // a warp's rows of the output are a box of dst
    cudaError_t e;
    dim3 grid((a.Tq * a.gqa + kTile - 1) / kTile, a.Hkv, a.B);   // packed (query, group head) rows per KV head
    // launch_inst is instantiated per kernel (the kernels share one function-pointer type, so a generic lambda would
    // share its "attribute set" flags between them)
    auto args = [&](auto launch) { e = launch(grid, smem, st, a, tmK, tmV, tmQ, tmO); };
    if constexpr (HD == 128) {
        // More than two full waves (of two CTAs per SM): CTAs that go on to the next tile themselves.  They ask for it when they start the one
        // before, so under a causal bound whoever has the longest tile also gets the longer of the second ones, which takes a third tile
        // to even out, and the more of them the longer the rows.  us, ordinary kernel / this one, F32 queries: 600 tiles of up to 96 keys
        // 25.4 / 24.6, 480 keys 32.3 / 29.5, 1920 keys 53.7 / 57.4; 640 tiles of 1280 keys 45.9 / 43.6, 2560 keys 67.8 / 71.0; 680 of 5400
        // 123 / 131; 704 of 1400 52.7 / 50.4; 752 of 12000 286 / 312; 768 of 3072 89.2 / 86.1; 960 of 5000 165 / 163.  Not causal, 600 tiles of
        // 128, 384, 1920 keys 27.0, 36.5, 100.2 / 25.8, 35.8, 98.6 (F16 queries 21.3, 33.0, 96.2 / 22.1, 32.8, 94.6).
        const long tiles = (long)grid.x * grid.y * grid.z;
        if (!a.has_mask && q_tma && o_tma && tiles > 4 * 148 + (a.causal && a.Lk > 1024 ? (a.Lk - 1024) / 16 : 0)) {
            const size_t smem_h128 = 1024 + (size_t)3 * TILE_BYTES + 112;
            static bool set[2][64] = {};
            auto go = [&](auto kern, bool (&smem_set)[64]) {
                cudaError_t e = set_smem_once(kern, smem_h128, smem_set);
                return e == cudaSuccess ? launch_pdl(kern, grid, kThreadsTc5, smem_h128, st, a, tmK, tmV, tmQ, tmO) : e;
            };
            e = q_tma == 2 ? go(fattn_prefill_tc5_h128_kernel<true>, set[0]) : go(fattn_prefill_tc5_h128_kernel<false>, set[1]);
            if (e == cudaSuccess) return B200_OK;
            snprintf(errbuf, errlen, "tcgen05 prefill launch: %s", cudaGetErrorString(e));
            return B200_E_CUDA;
        }
    }
    constexpr int QRAW = RAW_INST ? 2 : 0;
#define B200_GO(...) args(launch_inst<fattn_prefill_tc5_kernel<__VA_ARGS__>, FattnArgs, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap>)
    if (a.has_mask) {
        if (q_tma == 2) { if (o_tma) B200_GO(HD, NSTG, true, QRAW, true); else B200_GO(HD, NSTG, true, QRAW, false); }
        else if (q_tma == 1) { if (o_tma) B200_GO(HD, NSTG, true, 1, true); else B200_GO(HD, NSTG, true, 1, false); }
        else { if (o_tma) B200_GO(HD, NSTG, true, 0, true); else B200_GO(HD, NSTG, true, 0, false); }
    } else {
        if (q_tma == 2) { if (o_tma) B200_GO(HD, NSTG, false, QRAW, true); else B200_GO(HD, NSTG, false, QRAW, false); }
        else if (q_tma == 1) { if (o_tma) B200_GO(HD, NSTG, false, 1, true); else B200_GO(HD, NSTG, false, 1, false); }
        else { if (o_tma) B200_GO(HD, NSTG, false, 0, true); else B200_GO(HD, NSTG, false, 0, false); }
    }
#undef B200_GO
    if (e != cudaSuccess) {
        snprintf(errbuf, errlen, "tcgen05 prefill launch: %s", cudaGetErrorString(e));
        return B200_E_CUDA;
    }
    return B200_OK;
}

}  // namespace

bool tc5_supported(const FattnArgs& a) {
    if (a.hd != 64 && a.hd != 128) return false;
    if (a.k.type != B200_TYPE_F16 || a.v.type != B200_TYPE_F16) return false;
    if (!a.k.vec16 || !a.v.vec16) return false;
    if (a.softcap != 0.0f || a.n2 != 0) return false;
    if (!(a.scale > 0.0f)) return false;
    // explicit masks: any 2-byte aligned layout (rows that are not 16-byte aligned are read with 2-byte loads)
    if (a.relpos) {
        // fused bias: head_dim 128, F16 R with TMA-legal strides, no causal mask, bias rounded to F16
        if (a.hd != 128 || a.causal || a.relpos_f32) return false;
        if (a.scale < 0x1p-14f || a.scale > 0x1p13f) return false;   // (bias / scale goes into the score columns: far inside F32's range)
        if (a.r.type != B200_TYPE_F16 || !a.r.vec16 || a.r.nb1 <= 0 || a.r.nb2 <= 0) return false;
    }
    const int64_t lim = (int64_t)1 << 40;
    if (a.k.nb1 <= 0 || a.k.nb2 <= 0 || a.k.nb3 <= 0 || a.v.nb1 <= 0 || a.v.nb2 <= 0 || a.v.nb3 <= 0) return false;
    if (a.k.nb1 >= lim || a.k.nb2 >= lim || a.k.nb3 >= lim || a.v.nb1 >= lim || a.v.nb2 >= lim || a.v.nb3 >= lim) return false;
    return true;
}

int launch_prefill_tc5(const FattnArgs& a, cudaStream_t st, char* errbuf, size_t errlen) {
    if (a.relpos) return launch_relpos(a, st, errbuf, errlen);
    if (a.hd == 64) {
        const int n = a.has_mask ? 0 : h64_plan((long)((a.Tq * a.gqa + kTile - 1) / kTile) * a.Hkv * a.B, a.Lk, a.causal != 0);
        return n ? launch_h64(a, n, st, errbuf, errlen) : launch_t<64, 2>(a, st, errbuf, errlen);
    }
    return launch_t<128, 1>(a, st, errbuf, errlen);
}

int tc5_read_status(int* status) {
    int v = 0;
    const cudaError_t e = cudaMemcpyFromSymbol(&v, g_tc5_status, sizeof(int));
    if (e != cudaSuccess) return (int)e;
    *status = v;
    return 0;
}

int tc5_reset_status() {
    const int zero = 0;
    return (int)cudaMemcpyToSymbol(g_tc5_status, &zero, sizeof(int));
}

}  // namespace b200
