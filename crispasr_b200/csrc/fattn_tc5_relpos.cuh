// fattn_tc5_relpos.cuh — prefill with a relative-position bias (FastConformer, head_dim 128):
// logits = scale * Q_u.K^T + f16(scale * relshift(Q_v.R^T)), for one 128-row query tile of one (head, batch entry) per CTA.
//
// The bias of (query i, key J) is X[i][J - i + 127], X = Q_v . R_band^T with R_band row 0 = R row (Tq - 1) - q0 - 127: one more
// matrix product, whose columns have to be shifted by a different amount in every row.  A tcgen05.ld reads the same columns
// for all lanes, so the shift goes through shared memory:
//
//   four warps take the blocks of 64 X columns out of tensor memory as they are produced, each element once, round scale * x to F16 (where
//   the reference rounds, src/core/fastconformer.h:918) and store it at its key's place in a ring [128 query rows][4 panels of 64 keys].
//   A tile of 128 keys that is complete goes back, divided by scale, into the columns of its score tile, and the score product
//   adds to them.  The softmax warps then see finished scores, and their loop is that of a call without a bias.
//
// A row of the ring is written and read by one thread.  An infinite bias or a NaN stays with its own key, and what the table holds for keys
// at or beyond kv_len goes no further than the score columns that the softmax warps overwrite.
//
// Tile row r holds query 4 * (r % 32) + r / 32 of the tile: the rows of a warp differ by multiples of four keys, and a warp that
// starts its TMEM columns at 3 - (r / 32) has every group of four values on an 8-byte boundary of its row, whatever the lane.
// (With neighbouring queries in neighbouring lanes every row went through a bounce buffer and back, shifted by 2 bytes where needed.)
//
//   warps 0-7   softmax, epilogue: thread (r, ch) owns columns [64 ch, + 64) of tile row r (TMEM lane r)
//   warps 8-11  bias, as above; Q_v into tensor memory
//   warp  12    copies of K and V
//   warp  13    TMEM allocation; S products
//   warp  14    copies of R, X products
//   warp  15    P.V products
//   TMEM       [0,128) [128,256) S of even and odd tiles, P as f16x2 over the first 64 of its columns; [256,384) O; [384,448) X;
//              [448,512) the Q_v tile, f16x2
// Key tiles of 128: tile t takes X blocks 2t .. 2t + 3 and its bias is complete when the last of them is stored.  Scores run two tiles,
// the bias one tile ahead of the softmax.
//
// Relative error (2-norm) against 64 bits with the operator's own rounding of the bias: 8 ragged utterances of 138 frames 1.64e-4, 1500 frames
// 2.04e-4, 2500 frames 2.05e-4, 7500 frames 2.06e-4, the figures of a kernel that adds the rounded bias in its softmax warps.  The bias as an
// operand of the tensor cores, times 1 / scale as an F16 number in an identity matrix, is not that value: rounded as x * scale / d, d being that
// number, 2.5e-4, 3.2e-4, 3.3e-4, 3.5e-4, growing with the bias, and a NaN reaches the other keys of its product (2 x 7500 frames 645 us).
//
// 2 recordings of 7500 frames, bias added by the softmax warps / here: 873 -> 730 us in a burst, 953 -> 834 in a long run at the 1000 W limit; one
// of 1000 frames 24.9 -> 21.6, 8 utterances of up to 138 13.0 -> 12.6, a mask over 3000 frames 189 -> 130; of 5 frames 8.5 -> 8.6.
// What bounds it: 128 x 128 scores take 3.3 k clk, the softmax warps 2.5 k of them (exponentials 1.5 k, where the exponential unit needs 1.0 k;
// the meeting of the two warps of a row, the P store and the wait for the next scores the rest).  The columns of a score tile are free again 3 k
// clk after its P is there (P.V, bias, S and three hand-offs), and a block of X, of which a tile takes two, comes 1.5 k clk after the one
// before it has left its columns.  So the bias of a tile waits for P.V with the next block of X already taken out and its successor on the
// way (745 us before the blocks that nothing needs were left out; waiting ahead of that block 790, and with a wait of its own for the upper
// columns, which P leaves earlier, 837).
// Instruction fetch counts: five kinds of warps that each run straight-line code once per tile.
constexpr int kThreadsRelpos = 512;
constexpr int kRelBlock = 64;                          // X columns per step
constexpr int kRelRSlots = 4;                          // R blocks in flight
constexpr int kRelRBytes = kRelBlock * 2 * 128;        // 64 rows x 128 halves
constexpr int kRelTile = 2 * kPanelBytes;              // 128 rows x 128 halves
constexpr int kRelRingOff = kRelTile, kRelKOff = kRelRingOff + 2 * kRelTile, kRelVOff = kRelKOff + kRelTile, kRelROff = kRelVOff + kRelTile,
              kRelBarOff = kRelROff + kRelRSlots * kRelRBytes, kRelMiscOff = kRelBarOff + 24 * 8;
constexpr size_t kRelSmem = 1024 + (size_t)kRelMiscOff + 16 + 64 + 2 * kTile * sizeof(float);
static_assert(kRelSmem <= 232448, "shared memory of a CTA");

// Tile row of query i of the tile.
__device__ __forceinline__ int relpos_row(int i) { return ((i & 3) << 5) | (i >> 2); }

// 128-element query rows -> swizzled f16 operand tiles, 16 rows per warp, a warp instruction covers whole rows: lane l reads
// float4 l of one F32 row, or 16 bytes l % 16 of two F16 rows; all loads in flight at once.  BIAS: two tiles from one read,
// Q + bias_u and Q + bias_v, sums formed in fp32 and rounded once.  Rows at or beyond `rows` (of the tile) are zero.
template <bool F16, bool BIAS>
__device__ __forceinline__ void load_relpos_q(uint8_t* tile_u, uint8_t* tile_v, const uint8_t* base, int64_t nb1, int q0, int rows, const float* bias_u,
                                              const float* bias_v, int warp, int lane) {
    constexpr int N = F16 ? 8 : 4, RPI = F16 ? 2 : 1, K = 16 / RPI;   // elements per lane; rows per instruction; instructions
    const int c = (F16 ? lane & 15 : lane) * N;
    float bu[N], bv[N];
    if (BIAS) {
#pragma unroll
        for (int i = 0; i < N; i += 4) {
            const float4 x = load_global(reinterpret_cast<const float4*>(bias_u + c + i)), y = load_global(reinterpret_cast<const float4*>(bias_v + c + i));
            bu[i] = x.x, bu[i + 1] = x.y, bu[i + 2] = x.z, bu[i + 3] = x.w;
            bv[i] = y.x, bv[i + 1] = y.y, bv[i + 2] = y.z, bv[i + 3] = y.w;
        }
    }
    uint4 v[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int r = warp * 16 + k * RPI + (F16 ? lane >> 4 : 0);
        v[k] = make_uint4(0u, 0u, 0u, 0u);
        if (r < rows) v[k] = load_global(reinterpret_cast<const uint4*>(base + (int64_t)(q0 + r) * nb1 + c * (F16 ? 2 : 4)));
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int r = warp * 16 + k * RPI + (F16 ? lane >> 4 : 0), tr = relpos_row(r);
        const uint32_t off = (c >> 6) * kPanelBytes + tr * 128 + ((((c & 63) >> 3) ^ (tr & 7)) << 4) + (c & 4) * 2;
        float f[N];
        const uint32_t w[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (F16) {
                const float2 p = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
                f[(2 * i) % N] = p.x, f[(2 * i + 1) % N] = p.y;
            } else {
                f[i] = __uint_as_float(w[i]);
            }
        }
#pragma unroll
        for (int t = 0; t < (BIAS ? 2 : 1); t++) {
            uint32_t o[N / 2];
#pragma unroll
            for (int i = 0; i < N; i += 2) {
                const float x = BIAS && r < rows ? __fadd_rn(f[i], t ? bv[i] : bu[i]) : f[i];
                const float y = BIAS && r < rows ? __fadd_rn(f[i + 1], t ? bv[i + 1] : bu[i + 1]) : f[i + 1];
                o[i >> 1] = pack_half2(x, y);
            }
            uint8_t* p = (t ? tile_v : tile_u) + off;
            if constexpr (F16) *reinterpret_cast<uint4*>(p) = make_uint4(o[0], o[1], o[2 % (N / 2)], o[3 % (N / 2)]);
            else *reinterpret_cast<uint2*>(p) = make_uint2(o[0], o[1]);
        }
    }
}

// 32 bytes of one row per lane: whole sectors without a staging pass through shared memory (`wide`: 32-byte aligned rows).
__device__ __forceinline__ void store8(float* p, const uint32_t* r, float f, bool wide) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]) * f;
    if (wide) {
        asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]),
                     "f"(v[6]), "f"(v[7])
                     : "memory");
    } else {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}

// 64 mask values of a row as 32 pairs; those at or beyond `avail` (the end of the mask row) read as 0 and are never touched.  `align` is
// what the start and the strides of the mask are multiples of: one answer for all rows, so that the warp stays together, which the tensor
// memory instructions behind these loads need.  (load_global: an assembly load that is not volatile may be executed ahead of the test of
// its alignment.)  A warp load of 32 rows occupies L1 32 times whatever its width, and what shared memory leaves of L1 does not hold
// the tile's rows: rows on no 16-byte boundary are read as the nine 16-byte words around them and shifted into place, unless some of those
// reach beyond the mask [lo, hi) (4 x 1501 frames 307 -> 134 us, 11 utterances of up to 246 frames 47.8 -> 37.3, by 4- and 2-byte loads before; the
// aligned form as a block of its own 2 x 3000 frames 245 -> 200; all with the bias as an operand of the tensor cores; now the first takes 145).
__device__ __forceinline__ void load_mask_row(uint32_t (&mv)[32], const uint8_t* mptr, int avail, int align, const uint8_t* lo, const uint8_t* hi) {
    const uint32_t skew = (uint32_t)reinterpret_cast<uintptr_t>(mptr) & 15u;
    if (align >= 16 && avail >= 64) {
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const uint4 v = load_global(reinterpret_cast<const uint4*>(mptr) + q);
            mv[4 * q] = v.x, mv[4 * q + 1] = v.y, mv[4 * q + 2] = v.z, mv[4 * q + 3] = v.w;
        }
        return;
    }
    if (avail >= 64 && __all_sync(0xffffffffu, mptr - skew >= lo && mptr - skew + 144 <= hi)) {
        uint32_t w[36];
#pragma unroll
        for (int q = 0; q < 9; q++) {
            const uint4 v = load_global(reinterpret_cast<const uint4*>(mptr - skew) + q);
            w[4 * q] = v.x, w[4 * q + 1] = v.y, w[4 * q + 2] = v.z, w[4 * q + 3] = v.w;
        }
#pragma unroll
        for (int i = 0; i < 34; i++) w[i] = skew & 8u ? w[i + 2] : w[i];
#pragma unroll
        for (int i = 0; i < 33; i++) w[i] = skew & 4u ? w[i + 1] : w[i];
#pragma unroll
        for (int i = 0; i < 32; i++) mv[i] = __funnelshift_r(w[i], w[i + 1], (skew & 2u) * 8u);
        return;
    }
#pragma unroll
    for (int g = 0; g < 8; g++) {   // 16 bytes each
        const uint8_t* p = mptr + g * 16;
        uint32_t* m = mv + g * 4;
        if (avail >= g * 8 + 8 && align >= 16) {
            const uint4 v = load_global(reinterpret_cast<const uint4*>(p));
            m[0] = v.x, m[1] = v.y, m[2] = v.z, m[3] = v.w;
        } else if (avail >= g * 8 + 8 && align >= 4) {
#pragma unroll
            for (int i = 0; i < 4; i++) m[i] = load_global(reinterpret_cast<const uint32_t*>(p + i * 4));
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t l = g * 8 + 2 * i < avail ? load_global(reinterpret_cast<const uint16_t*>(p + i * 4)) : (uint16_t)0;
                const uint32_t h = g * 8 + 2 * i + 1 < avail ? load_global(reinterpret_cast<const uint16_t*>(p + i * 4 + 2)) : (uint16_t)0;
                m[i] = l | (h << 16);
            }
        }
    }
}

// Three barriers at once (a test takes 120 clocks or more to come back, also of a phase that is complete).
__device__ __forceinline__ bool mbar_wait_all(uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, uint32_t b2, uint32_t p2, volatile int* abort_flag) {
    const uint32_t t0 = mbar_test(b0, p0), t1 = mbar_test(b1, p1), t2 = mbar_test(b2, p2);
    return (t0 || mbar_wait(b0, p0, abort_flag)) && (t1 || mbar_wait(b1, p1, abort_flag)) && (t2 || mbar_wait(b2, p2, abort_flag));
}

template <bool HASMASK>
__global__ void __launch_bounds__(kThreadsRelpos, 1)
fattn_prefill_tc5_relpos_kernel(const FattnArgs a, const float inv_scale, const __grid_constant__ CUtensorMap tmK,
                                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmR) {
    constexpr int HD = 128;
    constexpr uint32_t IDESC_S = idesc_f16(kTile, false), IDESC_X = idesc_f16(kRelBlock, false), IDESC_PV = idesc_f16(HD, true);

    extern __shared__ uint8_t smem_dyn[];
    const uint32_t smem_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_dyn + (smem_base - smem_u32(smem_dyn));
    const uint32_t sQ = smem_base, sK = smem_base + kRelKOff, sV = smem_base + kRelVOff, sR = smem_base + kRelROff,
                   sBar = smem_base + kRelBarOff;
    const uint32_t bar_k_full = sBar /* [2]: halves of the head dimension */, bar_k_empty = sBar + 16 /* [2] */, bar_v_full = sBar + 32,
                   bar_v_empty = sBar + 40, bar_r_full = sBar + 48 /* [4] */, bar_s_full = sBar + 80 /* [2] */, bar_p_ready = sBar + 96 /* [2] */,
                   bar_o_done = sBar + 112, bar_x_full = sBar + 120, bar_x_free = sBar + 128, bar_b_full = sBar + 136 /* [2] */,
                   bar_qv = sBar + 152, bar_drain = sBar + 160 /* [2] */, bar_pv = sBar + 176 /* [2]: P.V of even and odd tiles */;
    uint8_t* misc = smem_gen + kRelMiscOff;
    volatile uint32_t* s_tmem_base = reinterpret_cast<volatile uint32_t*>(misc);
    volatile int* s_abort = reinterpret_cast<volatile int*>(misc + 4);
    volatile uint32_t* s_flag = reinterpret_cast<volatile uint32_t*>(misc + 16);   // [2][8]: one word of each softmax warp
    volatile float* s_row = reinterpret_cast<volatile float*>(misc + 80);          // [2][128]: maxima or sums of half rows

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int q0 = blockIdx.x * kTile, h = blockIdx.y, b = blockIdx.z;
    const int hk = h / a.gqa, bk = b / a.bq;
    const int rb3 = a.r_ne3 > 1 ? b : 0;
    if (tid == 14 * 32) {
        for (int i = 0; i < 24; i++) {
            const uint32_t bar = sBar + 8 * i;
            // one arrival per warp of the softmax or the bias group (P and the bias have a barrier for each of the two score tiles: a warp may be
            // a tile ahead of another one)
            const bool four = bar == bar_x_free || bar == bar_b_full || bar == bar_b_full + 8 || bar == bar_qv;
            mbar_init(bar, bar == bar_p_ready || bar == bar_p_ready + 8 ? 8 : (four ? 4 : 1));
        }
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmK)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmV)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmR)) : "memory");
    }
    // launched with programmatic stream serialisation: nothing is read before the previous kernel has completed
    const uint32_t behind_wait = wait_for_predecessors();

    int len_b = a.Lk;
    if (a.kv_len) {
        const int v = a.kv_len[b];
        len_b = v < 0 ? 0 : (v > a.Lk ? a.Lk : v);
    }
    const int tq_b = q_rows_of(a, b);   // query rows at or beyond it are padding of a batched launch: zeros
    const int n_tiles = (len_b > 0 && q0 < tq_b) ? (len_b + kTile - 1) / kTile : 0;
    if (n_tiles == 0) {
        if (tid < kTile && q0 + tid < a.Tq) {
            float4* out = reinterpret_cast<float4*>(a.dst + (((int64_t)b * a.Tq + q0 + tid) * a.dst_heads + h) * HD);
#pragma unroll
            for (int i = 0; i < HD / 4; i++) out[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        return;
    }
    // X blocks: 2 n_tiles + 2, but for the first one, which only rows from 64 on need (J - i + 127 < 64 with J >= 0), and the last one, which only
    // keys of the last tile from 64 on need, where there are none.  They are numbered from the first one taken, block m0; what the
    // ring holds in the places left out goes to dead rows and keys.
    const int m0 = tq_b - q0 <= 64 ? 1 : 0;
    const int n_blocks = 2 * n_tiles + (len_b - (n_tiles - 1) * kTile <= 64 ? 1 : 2) - m0;
    const int rb0 = a.Tq - 1 - q0 - 127 + kRelBlock * m0;  // R row of the first block's first column (may be negative: the copies fill with zeros)

    auto load_r = [&](int m) {
        const uint32_t bar = bar_r_full + 8 * (m & (kRelRSlots - 1)), dst = sR + (m & (kRelRSlots - 1)) * kRelRBytes;
        mbar_arrive_expect_tx(bar, kRelRBytes);
        tma_load_4d(dst, &tmR, bar, 0, rb0 + kRelBlock * m, h, rb3);
        tma_load_4d(dst + kRelRBytes / 2, &tmR, bar, 64, rb0 + kRelBlock * m, h, rb3);
    };
    auto load_k = [&](int j, int p) {
        mbar_arrive_expect_tx(bar_k_full + 8 * p, kPanelBytes);
        tma_load_4d(sK + p * kPanelBytes, &tmK, bar_k_full + 8 * p, p * 64, j * kTile, hk, bk);
    };
    auto load_v = [&](int j) {
        mbar_arrive_expect_tx(bar_v_full, kRelTile);
        tma_load_4d(sV, &tmV, bar_v_full, 0, j * kTile, hk, bk);
        tma_load_4d(sV + kPanelBytes, &tmV, bar_v_full, 64, j * kTile, hk, bk);
    };

    // ---- set-up ----
    if (tid == 14 * 32) {   // (the thread that set the barriers up)
#pragma unroll 1
        for (int m = 0; m < min(kRelRSlots, n_blocks); m++) load_r(m);
        load_k(0, 0);
        load_k(0, 1);
        load_v(0);
    }
    if (warp == 13) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(const_cast<uint32_t*>(s_tmem_base))),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (warp < 8) {
        // Q_u and Q_v tiles -> shared memory, Q_v into the ring, which is free until it is in tensor memory.  Aligned rows: warp w takes
        // rows [16w, 16w + 16) whole (load_relpos_q); with the position biases folded in, one read of Q serves both tiles.
        const uint8_t* q_base = a.q.p + (int64_t)h * a.q.nb2 + (int64_t)b * a.q.nb3;
        const uint8_t* qv_base = a.qv.p + (int64_t)h * a.qv.nb2 + (int64_t)b * a.qv.nb3;
        const int rows = a.Tq - q0;
        uint8_t *tu = smem_gen, *tv = smem_gen + kRelRingOff;
        if (a.bias_u != nullptr && a.q.vec16 && ((reinterpret_cast<uintptr_t>(a.bias_u) | reinterpret_cast<uintptr_t>(a.bias_v)) & 15) == 0) {
            if (a.q.type == B200_TYPE_F32) load_relpos_q<false, true>(tu, tv, q_base, a.q.nb1, q0, rows, a.bias_u + h * HD, a.bias_v + h * HD, warp, lane);
            else load_relpos_q<true, true>(tu, tv, q_base, a.q.nb1, q0, rows, a.bias_u + h * HD, a.bias_v + h * HD, warp, lane);
        } else if (a.bias_u == nullptr && a.q.vec16 && a.qv.vec16) {
            if (a.q.type == B200_TYPE_F32) load_relpos_q<false, false>(tu, nullptr, q_base, a.q.nb1, q0, rows, nullptr, nullptr, warp, lane);
            else load_relpos_q<true, false>(tu, nullptr, q_base, a.q.nb1, q0, rows, nullptr, nullptr, warp, lane);
            if (a.qv.type == B200_TYPE_F32) load_relpos_q<false, false>(tv, nullptr, qv_base, a.qv.nb1, q0, rows, nullptr, nullptr, warp, lane);
            else load_relpos_q<true, false>(tv, nullptr, qv_base, a.qv.nb1, q0, rows, nullptr, nullptr, warp, lane);
        } else {
            const int i = tid & 127, ch = tid >> 7, r = relpos_row(i);
            const int iq = q0 + i;
#pragma unroll 1
            for (int which = 0; which < 2; which++) {
                const View& qv = which ? a.qv : a.q;
                const uint8_t* rowp = (which ? qv_base : q_base) + (int64_t)iq * qv.nb1;
                const float* bias = which ? a.bias_v : a.bias_u;
#pragma unroll 1
                for (int c = 0; c < HD / 16; c++) {
                    const int cc = ch * (HD / 16) + c;
                    uint4 v = make_uint4(0u, 0u, 0u, 0u);
                    if (iq < a.Tq) v = bias != nullptr ? load8_plus_bias_as_half(rowp, qv.type, cc * 8, qv.vec16 != 0, bias + h * HD + cc * 8)
                                                       : q_chunk(rowp, qv.type, cc * 8, qv.vec16 != 0);
                    *reinterpret_cast<uint4*>((which ? tv : tu) + r * 128 + (cc >> 3) * kPanelBytes + (((cc & 7) ^ (r & 7)) << 4)) = v;
                }
            }
        }
        fence_proxy_async();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // the next launch may become resident as this one's CTAs leave (not where it is likely a conversion again, whose CTAs take the room)
    if (!a.behind_cast) let_dependents_launch();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *s_tmem_base, 0);
    const uint32_t tmem_S = tmem_base, tmem_O = tmem_base + 256, tmem_X = tmem_base + 384, tmem_Qv = tmem_base + 448;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    constexpr uint32_t desc_hi = smem_desc_hi(1024);
    bool ok = true;

    if (warp == 12) {
        // ================= copies of K and V =================
        if (lane == 0) {
            int k_issued = 1, v_issued = 1;
            auto next_k = [&](int j) {   // into the halves that S[j - 1] leaves
                for (int p = 0; p < 2 && ok; p++) {
                    ok = mbar_wait(bar_k_empty + 8 * p, (j - 1) & 1, s_abort);
                    if (ok) load_k(j, p);
                }
                if (ok) k_issued = j + 1;
            };
            if (n_tiles > 1) next_k(1);
            for (int j = 1; j < n_tiles && ok; j++) {
                if (j + 1 < n_tiles) next_k(j + 1);   // S[j] is issued ahead of P[j - 1].V[j - 1]
                if (ok) ok = mbar_wait(bar_v_empty, (j - 1) & 1, s_abort);
                if (!ok) break;
                load_v(j);
                v_issued = j + 1;
            }
            if (!ok) {   // drain: bounded waits for copies that may still be in flight (a half of K more than counted, too)
                for (int p = 0; p < 2; p++)
                    for (uint32_t it = 0; it < 4096 && !mbar_try_wait(bar_k_full + 8 * p, (k_issued - 1) & 1); ++it) __nanosleep(256);
                for (uint32_t it = 0; it < 4096 && !mbar_try_wait(bar_v_full, (v_issued - 1) & 1); ++it) __nanosleep(256);
                for (uint32_t it = 0; it < 4096; ++it) __nanosleep(64);
            }
        }
    } else if (warp == 13) {
        // ================= scores: Q_u.K^T onto the bias, two tiles ahead =================
        const uint32_t q_lo = smem_desc_lo(sQ, 16), k_lo = smem_desc_lo(sK, 16);
        for (int j = 0; j < n_tiles; j++) {
            const uint32_t s = tmem_S + (j & 1) * kTile;
            // K[j] is there, and the bias in the columns of S[j] (behind P[j - 2].V[j - 2], whose P lay in them)
            ok = warp_all(mbar_wait_all(bar_k_full, j & 1, bar_k_full + 8, j & 1, bar_b_full + 8 * (j & 1), (j >> 1) & 1, s_abort));
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < HD / 16; ks++) {
                    const uint32_t off16 = (uint32_t)(((ks >> 2) * kPanelBytes + (ks & 3) * 32) >> 4);
                    mma_ss(s, desc64(q_lo + off16, desc_hi), desc64(k_lo + off16, desc_hi), IDESC_S, 1u);
                    if (ks == 3) tc_commit(bar_k_empty);
                }
                tc_commit(bar_k_empty + 8);
                tc_commit(bar_s_full + 8 * (j & 1));
            }
            __syncwarp();
        }
        if (!ok) {   // no MMA of this warp may still be running when its memory is released
            if (elect_one()) tc_commit(bar_drain + 8);
            __syncwarp();
            for (uint32_t it = 0; it < 65536 && !mbar_try_wait(bar_drain + 8, 0); ++it) __nanosleep(256);
        }
        __syncwarp();
    } else if (warp == 15) {
        // ================= P.V products =================
        const uint32_t v_lo = smem_desc_lo(sV, kPanelBytes);
        for (int j = 0; j < n_tiles; j++) {
            ok = warp_all(mbar_wait_all(bar_v_full, j & 1, bar_p_ready + 8 * (j & 1), (j >> 1) & 1, bar_v_full, j & 1, s_abort));
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t p = tmem_S + (j & 1) * kTile;
                mma_ts(tmem_O, p, desc64(v_lo, desc_hi), IDESC_PV, j > 0 ? 1u : 0u);
#pragma unroll
                for (int ks = 1; ks < kTile / 16; ks++) mma_ts(tmem_O, p + ks * 8, desc64(v_lo + ks * (2048 >> 4), desc_hi), IDESC_PV, 1u);
                tc_commit(bar_pv + 8 * (j & 1));
                tc_commit(bar_v_empty);
                if (j + 1 == n_tiles) tc_commit(bar_o_done);
            }
            __syncwarp();
        }
        if (!ok) {
            if (elect_one()) tc_commit(bar_o_done);
            __syncwarp();
            for (uint32_t it = 0; it < 65536 && !mbar_try_wait(bar_o_done, 0); ++it) __nanosleep(256);
        }
        __syncwarp();
    } else if (warp == 14) {
        // ================= X products and copies of R =================
        const uint32_t r_lo = smem_desc_lo(sR, 16);
        int r_issued = min(kRelRSlots, n_blocks);
        ok = warp_all(mbar_wait(bar_qv, 0, s_abort));
        for (int m = 0; m < n_blocks && ok; m++) {
            ok = mbar_wait(bar_r_full + 8 * (m & (kRelRSlots - 1)), (m / kRelRSlots) & 1, s_abort) && (m == 0 || mbar_wait(bar_x_free, (m - 1) & 1, s_abort));
            ok = warp_all(ok);
            if (!ok) break;
            tc_fence_after();
            const bool more = m > 0 && m + kRelRSlots - 1 < n_blocks;
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < HD / 16; ks++)
                    mma_ts(tmem_X, tmem_Qv + ks * 8,
                           desc64(r_lo + (uint32_t)(((m & (kRelRSlots - 1)) * kRelRBytes + (ks >> 2) * (kRelRBytes / 2) + (ks & 3) * 32) >> 4), desc_hi), IDESC_X,
                           ks > 0 ? 1u : 0u);
                tc_commit(bar_x_full);
                if (more) load_r(m + kRelRSlots - 1);   // the slot of block m - 1, whose product has been read
            }
            __syncwarp();
            if (more) r_issued = m + kRelRSlots;
        }
        if (!ok) {
            if (elect_one()) tc_commit(bar_drain);
            __syncwarp();
            for (uint32_t it = 0; it < 65536 && !mbar_try_wait(bar_drain, 0); ++it) __nanosleep(256);
            for (int m = max(0, r_issued - kRelRSlots); m < r_issued; m++)
                for (uint32_t it = 0; it < 4096 && !mbar_try_wait(bar_r_full + 8 * (m & (kRelRSlots - 1)), (m / kRelRSlots) & 1); ++it) __nanosleep(256);
        }
        __syncwarp();
    } else if (warp >= 8) {
        // ================= bias: X columns to their keys =================
        const int w = warp & 3, r = tid & 127;
        uint8_t* const ring_row = smem_gen + kRelRingOff;
        {   // row r of the Q_v tile -> tensor memory (K elements 2c, 2c + 1 in column c)
            uint32_t x[2][32];
#pragma unroll
            for (int cc = 0; cc < HD / 8; cc++) {
                const uint4 v = *reinterpret_cast<const uint4*>(ring_row + (cc >> 3) * kPanelBytes + r * 128 + (((cc & 7) ^ (r & 7)) << 4));
                uint32_t* o = x[cc >> 3] + (cc & 7) * 4;
                o[0] = v.x, o[1] = v.y, o[2] = v.z, o[3] = v.w;
            }
            tmem_st32(tmem_Qv + lane_base, x[0]);
            tmem_st32(tmem_Qv + lane_base + 32, x[1]);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_qv);
        }
        // Group g (four keys) of block m belongs to key group 16 m + g + lane - 32, g = 0 being the values across the border of two
        // blocks.  Its byte in the ring: panel (m - 2 + (g + lane) / 16) % 4, then row r of the panel, swizzled.
        uint32_t off[16];
#pragma unroll
        for (int g = 0; g < 16; g++) {
            const uint32_t u = g + lane;
            off[g] = (2u + m0 + (u >> 4)) * kPanelBytes + r * 128 + ((((u >> 1) & 7) ^ (r & 7)) << 4) + (u & 1) * 8;
        }
        uint32_t carry[4] = {0u, 0u, 0u, 0u};
        const uint64_t scale2 = pack2(a.scale, a.scale), inv_scale2 = pack2(inv_scale, inv_scale);
        auto scaled = [&](float x0, float x1) {   // f16(scale * x), the reference's rounding
            unpack2(mul2(pack2(x0, x1), scale2), x0, x1);
            return cvt_f16x2(x0, x1);
        };
        // Tile t is complete with block 2t + 3.  Its columns of the score tile start from bias / scale; they are free once P[t - 2].V[t - 2], whose P
        // lies in them, has completed, which is awaited with the next block of X already out of tensor memory (not for the first two tiles).
        int m = 0, t = 0;
        while (t < n_tiles) {
            const bool complete = m0 + m >= 2 * t + 4 || m == n_blocks, block = m < n_blocks && !(complete && t < 2);
            uint32_t o[32], pv_there = 0;
            if (block) {
                ok = warp_all(mbar_wait(bar_x_full, m & 1, s_abort));   // (the tensor memory instructions want the warp together)
                if (!ok) break;
                tc_fence_after();
                uint32_t first[4], xa[32], xb[32];
                tmem_ld4(tmem_X + lane_base - 1 - w, first);         // (columns before the block's own are not used)
                tmem_ld32(tmem_X + lane_base + 3 - w, xa);
                tmem_ld32(tmem_X + lane_base + 35 - w, xb);          // (nor the last ones: they wait for the next block)
                tmem_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_x_free);
                if (complete) pv_there = mbar_test(bar_pv + 8 * (t & 1), ((t >> 1) - 1) & 1);
                {
                    float e[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) e[k] = __uint_as_float(k <= w ? carry[k] : first[k]);
                    o[0] = scaled(e[0], e[1]), o[1] = scaled(e[2], e[3]);
                }
#pragma unroll
                for (int i = 0; i < 32; i += 2) o[2 + (i >> 1)] = scaled(__uint_as_float(xa[i]), __uint_as_float(xa[i + 1]));
#pragma unroll
                for (int i = 0; i < 28; i += 2) o[18 + (i >> 1)] = scaled(__uint_as_float(xb[i]), __uint_as_float(xb[i + 1]));
#pragma unroll
                for (int k = 0; k < 4; k++) carry[k] = xb[28 + k];
            }
            if (complete) {
                if (t >= 2) {
                    ok = warp_all(pv_there || mbar_wait(bar_pv + 8 * (t & 1), ((t >> 1) - 1) & 1, s_abort));
                    if (!ok) break;
                    tc_fence_after();
                }
                const uint8_t* row = ring_row + (t & 1) * kRelTile + r * 128;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    uint32_t f[32];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const int cc = 4 * q + i;
                        const uint4 v = *reinterpret_cast<const uint4*>(row + (cc >> 3) * kPanelBytes + (((cc & 7) ^ (r & 7)) << 4));
                        const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&w4[k]));
                            float f0, f1;
                            unpack2(mul2(pack2(x.x, x.y), inv_scale2), f0, f1);
                            f[8 * i + 2 * k] = __float_as_uint(f0), f[8 * i + 2 * k + 1] = __float_as_uint(f1);
                        }
                    }
                    tmem_st32(tmem_S + (t & 1) * kTile + lane_base + q * 32, f);
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_b_full + 8 * (t & 1));
                t++;
            }
            if (block) {
#pragma unroll
                for (int g = 0; g < 16; g++) {
                    *reinterpret_cast<uint2*>(ring_row + (off[g] & (4 * kPanelBytes - 1))) = make_uint2(o[2 * g], o[2 * g + 1]);
                    off[g] += kPanelBytes;
                }
                m++;
            }
        }
    } else {
        // ================= softmax =================
        const int r = tid & 127, ch = tid >> 7, iq = q0 + 4 * lane + (warp & 3);
        const float c = a.scale * kLog2e;
        const uint64_t c2 = pack2(c, c), l2e2 = pack2(kLog2e, kLog2e);
        float m_ref = -INFINITY, l_run = 0.0f;
        // Explicit F16 mask added on top of the bias (bucket padding of src/canary_ctc.cpp:370-382, the local-attention
        // window of src/core/fastconformer.h:887-895): this thread's row of [Lk, Tq, 1|H, 1|B];
        // rows past Tq (the padding rows of the last query tile) read row 0.
        const uint8_t* mrow = HASMASK ? a.mask.p + behind_wait + (int64_t)(iq < a.Tq ? iq : 0) * a.mask.nb1 +
                                            (int64_t)(h % a.mask_ne2) * a.mask.nb2 + (int64_t)(b % a.mask_ne3) * a.mask.nb3 + ch * 128
                                      : nullptr;
        const uint32_t mask_bits = (uint32_t)(reinterpret_cast<uintptr_t>(a.mask.p) | a.mask.nb1 | a.mask.nb2 | a.mask.nb3);
        const int mask_align = (mask_bits & 15) == 0 ? 16 : ((mask_bits & 3) == 0 ? 4 : 2);
        const uint8_t* mask_end = a.mask.p + (int64_t)(a.mask_ne3 - 1) * a.mask.nb3 + (int64_t)(a.mask_ne2 - 1) * a.mask.nb2 + (int64_t)(a.Tq - 1) * a.mask.nb1 + (int64_t)a.Lk * 2;
        // The two warps of 32 rows meet at a hardware barrier (a fraction of an mbarrier's latency).  Both take part in every meeting, also when
        // a wait of theirs ran out: kFailed tells the other one, and both leave.
        constexpr uint32_t kFailed = 2u;
        uint32_t meeting = 0, s_there = 0;   // s_there: an early answer for the tile's scores, which have normally been there for long
        auto meet = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 3)) : "memory"); };
        auto either = [&](uint32_t mine) {   // one word of each warp, or-ed; two slots: a warp is never two meetings ahead
            if (lane == 0) s_flag[(meeting & 1) * 8 + warp] = mine;
            meet();
            const uint32_t both = mine | s_flag[(meeting & 1) * 8 + (warp ^ 4)];
            meeting++;
            return both;
        };
        auto other_half = [&](float v) {   // the value of the row's other thread
            s_row[ch * 128 + r] = v;
            meet();
            return s_row[(ch ^ 1) * 128 + r];
        };
        for (int j = 0; j < n_tiles; j++) {
            const uint32_t s_tile = tmem_S + (j & 1) * kTile + lane_base, s_cols = s_tile + ch * 64;
            const int n_valid = len_b - j * kTile - ch * 64;
            // P = exp2(S*c - m_ref) against a reference that need not be the maximum: the half row's sum bounds every P.  The maximum is
            // taken in the first tile and where a sum passes kRedoSumRelpos, which has O and l rescaled and P computed again.
            uint32_t pm[32];   // the mask, pair by pair replaced by P
            float lsum = 0.0f;
            bool take_max = j == 0, waited = false;
#pragma unroll 1
            for (;;) {
                if constexpr (HASMASK) load_mask_row(pm, mrow + (int64_t)j * kTile * 2, a.Lk - j * kTile - ch * 64, mask_align, a.mask.p, mask_end);
                if (!waited) {
                    ok = warp_all(s_there || mbar_wait(bar_s_full + 8 * (j & 1), (j >> 1) & 1, s_abort));
                    tc_fence_after();
                    waited = true;
                    if (n_valid < 64) {   // the last tile: -inf into the columns of keys that do not exist
#pragma unroll 1
                        for (int q = 0; q < 4; q++) {
                            uint32_t x[16];
                            tmem_ld16(s_cols + q * 16, x);
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 16; i++)
                                if (q * 16 + i >= n_valid) x[i] = 0xFF800000u;
                            tmem_st16(s_cols + q * 16, x);
                        }
                        tmem_wait_st();
                    }
                }
                // logits (log2 domain) of 16 columns, minus m
                auto logits = [&](uint32_t (&sx)[16], int col0, uint64_t nm2) {
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        uint64_t add = nm2;
                        if constexpr (HASMASK) {
                            const float2 m2 = __half22float2(*reinterpret_cast<const __half2*>(&pm[(col0 + i) >> 1]));
                            add = fma2(pack2(m2.x, m2.y), l2e2, nm2);
                        }
                        float t0, t1;
                        unpack2(fma2(pack2(__uint_as_float(sx[i]), __uint_as_float(sx[i + 1])), c2, add), t0, t1);
                        sx[i] = __float_as_uint(t0), sx[i + 1] = __float_as_uint(t1);
                    }
                };
                uint32_t sA[16], sB[16];
                if (take_max) {
                    float mx = -INFINITY;
#pragma unroll(HASMASK ? 4 : 1)
                    for (int q = 0; q < 4; q++) {
                        tmem_ld16(s_cols + q * 16, sA);
                        tmem_wait_ld();
                        logits(sA, q * 16, 0ull);
#pragma unroll
                        for (int i = 0; i < 16; i += 2) mx = max3(mx, __uint_as_float(sA[i]), __uint_as_float(sA[i + 1]));
                    }
                    const float m_new = fmaxf(m_ref, fmaxf(mx, other_half(mx)));
                    const float alpha = (m_ref == -INFINITY) ? 0.0f : ex2(m_ref - m_new);
                    l_run *= alpha;
                    if (j > 0 && ok) {
                        ok = warp_all(mbar_wait(bar_v_empty, (j - 1) & 1, s_abort));   // O is at rest: P[j-1].V[j-1] has completed
                        tc_fence_after();
#pragma unroll 1
                        for (int q4 = 0; q4 < 4; q4++) {
                            tmem_ld16(tmem_O + lane_base + ch * 64 + q4 * 16, sA);
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 16; i++) sA[i] = __float_as_uint(__uint_as_float(sA[i]) * alpha);
                            tmem_st16(tmem_O + lane_base + ch * 64 + q4 * 16, sA);
                        }
                    }
                    m_ref = m_new;
                }
                const float m_use = (m_ref == -INFINITY) ? kNoReference : m_ref;
                const uint64_t nm2 = pack2(-m_use, -m_use);
                uint64_t ls[2] = {0ull, 0ull};
                auto chunk = [&](uint32_t (&sx)[16], int col0) {
                    logits(sx, col0, nm2);
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        const float p0 = ex2(__uint_as_float(sx[i])), p1 = ex2(__uint_as_float(sx[i + 1]));
                        ls[(i >> 1) & 1] = add2(ls[(i >> 1) & 1], pack2(p0, p1));
                        pm[(col0 + i) >> 1] = cvt_f16x2(p0, p1);
                    }
                };
                // rolling chunks: the load of a chunk runs under the exponentials of the one before it
                tmem_ld16(s_cols, sA);
                tmem_ld16(s_cols + 16, sB);
                tmem_wait_ld();
                chunk(sA, 0);
                tmem_ld16(s_cols + 32, sA);
                chunk(sB, 16);
                tmem_wait_ld();
                tmem_ld16(s_cols + 48, sB);
                chunk(sA, 32);
                tmem_wait_ld();
                chunk(sB, 48);
                float l0, l1;
                unpack2(add2(ls[0], ls[1]), l0, l1);
                lsum = l0 + l1;
                // behind this meeting both warps have read their scores, which the P stores overwrite
                const uint32_t f = either((__any_sync(0xffffffffu, lsum > kRedoSumRelpos) ? 1u : 0u) | (ok ? 0u : kFailed));
                ok = !(f & kFailed);
                if (!ok || take_max || !f) break;
                take_max = true;
            }
            if (!ok) break;
            l_run += lsum;
            tmem_st32(s_tile + ch * 32, pm);
            s_there = mbar_test(bar_s_full + 8 * (~j & 1), ((j + 1) >> 1) & 1);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_p_ready + 8 * (j & 1));
        }
        const float l_tot = l_run + other_half(l_run), inv = l_tot > 0.0f ? 1.0f / l_tot : 0.0f;
        if (ok) ok = warp_all(mbar_wait(bar_o_done, 0, s_abort));
        if (ok) {   // (a failed wait has set the abort flag: the host reports it)
            tc_fence_after();
            float* out = a.dst + (((int64_t)b * a.Tq + iq) * a.dst_heads + h) * HD + ch * 64;
            const bool wide = (reinterpret_cast<uintptr_t>(a.dst) & 31) == 0;
#pragma unroll
            for (int q4 = 0; q4 < 2; q4++) {
                uint32_t oreg[32];
                tmem_ld32(tmem_O + lane_base + ch * 64 + q4 * 32, oreg);
                tmem_wait_ld();
                if (iq >= tq_b) {   // padding row of a batched launch: literal zeros
#pragma unroll
                    for (int i = 0; i < 32; i++) oreg[i] = 0u;
                }
                if (iq < a.Tq) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) store8(out + q4 * 32 + i, oreg + i, inv, wide);
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 13) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}
