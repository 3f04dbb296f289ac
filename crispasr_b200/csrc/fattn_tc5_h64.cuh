// fattn_tc5_h64.cuh — head_dim 64 prefill without an explicit mask: four CTAs per SM, 64 keys per step.
//
// The exponential unit bounds this path (16 ex2 per clock and SM: 1024 clk per 128 x 128 scores, against 512 clk of
// tensor work at head_dim 64), so the layout serves one aim: that on every scheduler some softmax warp always has
// exponentials to issue.  Between two score tiles a softmax warp waits for its own chain (P stored -> barrier -> the
// issuing thread -> 8 MMAs -> barrier -> TMEM load, about 1 k clk); with two CTAs per SM and 128-key tiles the unit idled
// 35-50 % of the time.  A 64-key tile needs 64 + 64 TMEM columns (P takes the score columns it came from), 48 KB of shared
// memory and 96 registers for 160 threads: four CTAs fit, and a chain of one is covered by 3 x 512 clk of exponentials of
// the other three.  The price is a score product with N = 64, whose A operand (the query tile) is read from shared memory
// twice as often: 384 instead of 256 clk per 128 x 128 scores, still below the exponentials.
//
//   warps 0-3  softmax / epilogue: thread r owns query row r (TMEM lane r)
//   warp  4    TMEM allocation; its lane 0 issues all tensor copies and all MMAs
//   TMEM       [0,64) S, P as f16x2 in [0,32); [64,128) O
// Per step j the issuing thread waits for P[j] (which also says that S[j] and, through the order of the tensor pipe,
// P[j-1].V[j-1] are complete), issues P[j].V[j] and S[j+1], then refills the K slot of S[j] and the V slot of step j - 1:
// no "slot empty" barriers exist.
//
// 64 windows of the large encoder (T = 1500): 1277 -> 917 us in a burst (577 -> 804 TFLOP/s, 0.56 of the sustained GEMM rate,
// 1.2 k clk per 128 x 128 scores); in a long run 1065-1080 us at the 1000 W limit, whose 1.59-1.65 GHz (1.9 GHz before) make
// that 1.4 k clk.
constexpr int kH64Keys = 64;
constexpr int kH64Threads = 160;
constexpr int kH64KvBytes = kH64Keys * 128;   // one K or V tile
constexpr size_t kH64Smem = 1024 + (size_t)kPanelBytes + 4 * kH64KvBytes + 8 * 8 + 16;

__device__ __forceinline__ uint32_t peer_smem(uint32_t addr, int rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    return remote;
}
__device__ __forceinline__ float4 ld_peer_v4(uint32_t p) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ float2 ld_peer_v2(uint32_t p) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(p) : "memory");
    return v;
}

// Every eighth pair of exponentials goes to the FMA pipe: 64 windows of the large encoder 1086 -> 1074 us, 8 windows 141.1 ->
// 139.4, four windows 74.5 -> 71.5; every fourth pair costs more issue slots (and power) than the unit's time it frees (990
// against 917 us in a burst).
constexpr int kH64PolyEvery = 8;

// QTMA: F16 query rows arrive by one tensor copy (else the softmax warps load and convert them); OTMA: the output leaves by
// tensor stores (else by the threads).  SPLIT: the CTAs of a cluster share one query tile, each takes a range of its key
// steps; at the end they leave their O rows and (m, l) in shared memory and each merges and writes a share of the rows.
// For launches with fewer tiles than the SMs can run at full pace (h64_plan): a lone CTA per SM spends 0.75 us per step,
// its own hand-off chain, which two CTAs per SM hide for each other and four CTAs fill.
template <bool QTMA, bool OTMA, bool SPLIT = false>
__global__ void __launch_bounds__(kH64Threads, 4)
fattn_prefill_tc5_h64_kernel(const FattnArgs a, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                             const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmO) {
    constexpr int HD = 64;
    constexpr uint32_t IDESC_S = idesc_f16(kH64Keys, false), IDESC_PV = idesc_f16(HD, true);
    extern __shared__ uint8_t smem_dyn[];
    const uint32_t smem_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_dyn + (smem_base - smem_u32(smem_dyn));
    const uint32_t sQ = smem_base, sK = sQ + kPanelBytes, sV = sK + 2 * kH64KvBytes, sBar = sV + 2 * kH64KvBytes;
    const uint32_t bar_k = sBar, bar_v = sBar + 16, bar_s_full = sBar + 32, bar_p_ready = sBar + 40, bar_o_done = sBar + 48, bar_q = sBar + 56;
    uint8_t* misc = smem_gen + kPanelBytes + 4 * kH64KvBytes + 64;
    volatile uint32_t* s_tmem_base = reinterpret_cast<volatile uint32_t*>(misc);
    volatile int* s_abort = reinterpret_cast<volatile int*>(misc + 4);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // launched with programmatic stream serialisation: but for the query prefetch below, nothing is read or written before the previous
    // kernel has completed
    constexpr bool kPrefetchQ = !QTMA && !SPLIT;
    if (!kPrefetchQ) asm volatile("griddepcontrol.wait;" ::: "memory");
    // tile order and GQA packing as in fattn_prefill_tc5_kernel
    const int n_split = SPLIT ? a.n_splits : 1, split = SPLIT ? (int)blockIdx.x % n_split : 0;
    int q0 = ((int)blockIdx.x / n_split) * kTile, hk = blockIdx.y, b = blockIdx.z;
    if (!SPLIT && a.causal) {
        const int lin = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z), hb = gridDim.y * gridDim.z;
        q0 = (gridDim.x - 1 - lin / hb) * kTile;
        hk = (lin % hb) % gridDim.y, b = (lin % hb) / gridDim.y;
    }
    // Behind a conversion of K and V, which lets this kernel become resident early, the query rows that the threads will load are brought
    // into L2 meanwhile: four windows of 20 heads, all F32, 89.1 -> 86.7 us per launch in a graph, ten of 500 frames 44.8 -> 42.2.  (Behind a kernel that
    // does not, and where a cluster shares a tile, it only delays: one window of 8 heads 17.0 -> 17.3.  For tiles that come by one copy
    // it measured nothing.)
    if (kPrefetchQ && a.behind_cast && warp < 4 && q0 + tid < a.Tq * a.gqa) {
        const uint8_t* rowp = a.q.p + (int64_t)((q0 + tid) / a.gqa) * a.q.nb1 + (int64_t)(hk * a.gqa + (q0 + tid) % a.gqa) * a.q.nb2 + (int64_t)b * a.q.nb3;
        prefetch_l2(rowp);
        if (a.q.type == B200_TYPE_F32) prefetch_l2(rowp + 128);
    }
    if (kPrefetchQ) asm volatile("griddepcontrol.wait;" ::: "memory");
    const int bk = b / a.bq;
    const int rows_total = a.Tq * a.gqa;
    const int tq_b = q_rows_of(a, b);
    const int rows_live = tq_b * a.gqa;
    int len_b = a.Lk;
    if (a.kv_len) {
        const int v = a.kv_len[b];
        len_b = v < 0 ? 0 : (v > a.Lk ? a.Lk : v);
    }
    const int n_past = n_past_of(a, len_b, tq_b);
    int kmax = q0 < rows_live ? len_b : 0;
    if (a.causal) kmax = min(kmax, n_past + min((q0 + kTile - 1) / a.gqa + 1, tq_b));
    const int n_all = kmax > 0 ? (kmax + kH64Keys - 1) / kH64Keys : 0;
    const int tps = (n_all + n_split - 1) / n_split, t0 = split * tps;   // this CTA's steps: [t0, t0 + n_tiles)
    const int n_tiles = SPLIT ? max(0, min(n_all - t0, tps)) : n_all;
    if (n_all == 0) {  // nothing to attend to: zeros
        if (split == 0 && tid < kTile && q0 + tid < rows_total) {
            const int iq = (q0 + tid) / a.gqa, h = hk * a.gqa + (q0 + tid) % a.gqa;
            float4* out = reinterpret_cast<float4*>(a.dst + (((int64_t)b * a.Tq + iq) * a.dst_heads + h) * HD);
#pragma unroll
            for (int i = 0; i < HD / 4; i++) out[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        return;
    }

    auto load_k = [&](int j) {
        const uint32_t bar = bar_k + 8 * (j & 1);
        mbar_arrive_expect_tx(bar, kH64KvBytes);
        tma_load_4d(sK + (j & 1) * kH64KvBytes, &tmK, bar, 0, (t0 + j) * kH64Keys, hk, bk);
    };
    auto load_v = [&](int j) {
        const uint32_t bar = bar_v + 8 * (j & 1);
        mbar_arrive_expect_tx(bar, kH64KvBytes);
        tma_load_4d(sV + (j & 1) * kH64KvBytes, &tmV, bar, 0, (t0 + j) * kH64Keys, hk, bk);
    };
    if (warp == 4) {
        if (lane == 0) {
            for (int i = 0; i < 8; i++) mbar_init(sBar + 8 * i, sBar + 8 * i == bar_p_ready ? 4 : 1);   // P: one arrival per softmax warp
            *s_abort = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            if (!SPLIT || n_tiles > 0) {
                if (QTMA) {
                    mbar_arrive_expect_tx(bar_q, kPanelBytes);
                    tma_load_4d(sQ, &tmQ, bar_q, 0, hk * a.gqa, q0 / a.gqa, b);
                }
                load_k(0);
                load_v(0);
            }
            if (n_tiles > 1) load_k(1);
        }
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(const_cast<uint32_t*>(s_tmem_base))),
                     "r"(128u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    } else if (!QTMA) {
        const int iq = (q0 + tid) / a.gqa, h = hk * a.gqa + (q0 + tid) % a.gqa;
        const uint8_t* rowp = a.q.p + (int64_t)iq * a.q.nb1 + (int64_t)h * a.q.nb2 + (int64_t)b * a.q.nb3;
        if (a.q.type == B200_TYPE_F32 && a.q.vec16) load_q_rows_f32_coalesced<HD>(smem_gen, warp, lane, q0 + tid < rows_total ? rowp : nullptr);
        else if (a.q.type == B200_TYPE_F16 && a.q.vec16) load_q_rows_f16_coalesced<HD>(smem_gen, warp, lane, q0 + tid < rows_total ? rowp : nullptr);
        else load_q_row<HD>(smem_gen, tid, rowp, a.q.type, a.q.vec16 != 0, q0 + tid < rows_total);
        fence_proxy_async();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // The next launch (the next layer's) may become resident as this one's CTAs leave: three windows of 12 heads, 700 frames, 15.9 -> 15.4
    // us per launch.  Not where the next one is likely a conversion again: its CTAs take the room of the attention's (44 -> 46 us).
    if (!a.behind_cast) let_dependents_launch();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *s_tmem_base, 0);
    const uint32_t tmem_S = tmem_base, tmem_P = tmem_base, tmem_O = tmem_base + 64;

    if (warp == 4) {
        // ================= copies and MMAs =================
        {
            const uint32_t q_lo = smem_desc_lo(sQ, 16), k_lo = smem_desc_lo(sK, 16), v_lo = smem_desc_lo(sV, kPanelBytes);
            constexpr uint32_t desc_hi = smem_desc_hi(1024);
            auto issue_s = [&](int j) {
                const uint32_t kd = k_lo + (j & 1) * (kH64KvBytes >> 4);
#pragma unroll
                for (int ks = 0; ks < HD / 16; ks++)
                    mma_ss(tmem_S, desc64(q_lo + ks * 2, desc_hi), desc64(kd + ks * 2, desc_hi), IDESC_S, ks > 0 ? 1u : 0u);
                tc_commit(bar_s_full);
            };
            int k_issued = min(2, n_tiles), v_issued = 1;
            const bool any = !SPLIT || n_tiles > 0;   // a split beyond the last step has nothing to do
            bool ok = !any || ((!QTMA || mbar_wait(bar_q, 0, s_abort)) && mbar_wait(bar_k, 0, s_abort));
            ok = warp_all(ok);
            if (ok && any) {
                tc_fence_after();
                if (elect_one()) {
                    issue_s(0);
                    if (n_tiles > 1) load_v(1);
                }
                v_issued = min(2, n_tiles);
            }
            for (int j = 0; j < n_tiles && ok; j++) {
                const bool more = j + 1 < n_tiles;
                ok = mbar_wait(bar_v + 8 * (j & 1), (j >> 1) & 1, s_abort);
                if (ok && more) ok = mbar_wait(bar_k + 8 * ((j + 1) & 1), ((j + 1) >> 1) & 1, s_abort);
                if (ok) ok = mbar_wait(bar_p_ready, j & 1, s_abort);
                ok = warp_all(ok);
                if (!ok) break;
                tc_fence_after();
                const uint32_t vd = v_lo + (j & 1) * (kH64KvBytes >> 4);
                if (elect_one()) {
                    mma_ts(tmem_O, tmem_P, desc64(vd, desc_hi), IDESC_PV, j > 0 ? 1u : 0u);
#pragma unroll
                    for (int ks = 1; ks < kH64Keys / 16; ks++) mma_ts(tmem_O, tmem_P + ks * 8, desc64(vd + ks * (2048 >> 4), desc_hi), IDESC_PV, 1u);
                    if (more) issue_s(j + 1);
                    else tc_commit(bar_o_done);
                    if (j > 0 && more) load_v(j + 1);       // the slot of P[j-1].V[j-1]
                    if (j + 2 < n_tiles) load_k(j + 2);   // the slot of S[j]
                }
                __syncwarp();
                if (j > 0 && more) v_issued = j + 2;
                if (j + 2 < n_tiles) k_issued = j + 3;
            }
            if (!ok) {
                // no MMA and no copy of this CTA may still be running when its memory is released (the commit comes from the
                // lane that issued the MMAs)
                if (elect_one()) tc_commit(bar_o_done);
                __syncwarp();
                for (uint32_t it = 0; it < 65536 && !mbar_try_wait(bar_o_done, 0); ++it) __nanosleep(256);
                if (QTMA)
                    for (uint32_t it = 0; it < 4096 && !mbar_try_wait(bar_q, 0); ++it) __nanosleep(256);
                for (int j = max(0, k_issued - 2); j < k_issued; j++)
                    for (uint32_t it = 0; it < 4096 && !mbar_try_wait(bar_k + 8 * (j & 1), (j >> 1) & 1); ++it) __nanosleep(256);
                for (int j = max(0, v_issued - 2); j < v_issued; j++)
                    for (uint32_t it = 0; it < 4096 && !mbar_try_wait(bar_v + 8 * (j & 1), (j >> 1) & 1); ++it) __nanosleep(256);
            }
            __syncwarp();
        }
    } else {
        // ================= softmax / epilogue =================
        const int r = tid;
        const bool row_live = q0 + r < rows_live;
        const int iq_dst = (q0 + r) / a.gqa, h = hk * a.gqa + (q0 + r) % a.gqa;
        const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
        const float c = a.scale * kLog2e;
        int kend = len_b;
        if (a.causal) kend = min(kend, n_past + (row_live ? iq_dst : a.Tq) + 1);
        float m_ref = -INFINITY, l_run = 0.0f;
        const uint64_t c2 = pack2(c, c);
        bool ok = true;
        auto step_max = [&](int n_valid) {   // maximum of this row's scores of the step
            float mx = -INFINITY;
#pragma unroll 1
            for (int half = 0; half < 2; half++) {
                uint32_t x[32];
                tmem_ld32(tmem_S + lane_base + half * 32, x);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; i += 2)
                    mx = max3(mx, half * 32 + i < n_valid ? __uint_as_float(x[i]) : -INFINITY, half * 32 + i + 1 < n_valid ? __uint_as_float(x[i + 1]) : -INFINITY);
            }
            return mx;
        };
        for (int j = 0; j < n_tiles; j++) {
            ok = mbar_wait(bar_s_full, j & 1, s_abort);
            if (!ok) break;
            tc_fence_after();
            const int n_valid = kend - (t0 + j) * kH64Keys;   // columns >= n_valid of this row are masked
            const bool full_tile = __all_sync(0xffffffffu, n_valid >= kH64Keys);
            if (j == 0) {   // a first reference: the maximum of the row's first 32 scores (the check below corrects it)
                uint32_t x[32];
                tmem_ld32(tmem_S + lane_base, x);
                tmem_wait_ld();
                float mx = -INFINITY;
#pragma unroll
                for (int i = 0; i < 32; i += 2) mx = max3(mx, i < n_valid ? __uint_as_float(x[i]) : -INFINITY, i + 1 < n_valid ? __uint_as_float(x[i + 1]) : -INFINITY);
                m_ref = mx * c;
            }
            uint32_t preg[32];
            float lsum = 0.0f;
            // P = exp2(S*c - m_ref) against a reference that need not be the maximum: the step's row sum (needed anyway) bounds
            // every P of the row.  No running maximum is kept - one instruction in six of this loop; only a row whose sum passes
            // kRedoSum has the step's maximum taken, O and l rescaled and P redone (947 -> 925 us at 64 windows).
            for (int attempt = 0; attempt < 2; attempt++) {
                const float m_use = (m_ref == -INFINITY) ? kNoReference : m_ref;
                uint64_t ls2[2] = {0ull, 0ull};
                const uint64_t nm2 = pack2(-m_use, -m_use);
                uint32_t sA[16], sB[16];
                auto chunk = [&](uint32_t (&sx)[16], uint32_t* p8, int col0) {
                    if (!full_tile) {
                        if (__all_sync(0xffffffffu, col0 >= n_valid)) {
#pragma unroll
                            for (int i = 0; i < 8; i++) p8[i] = 0u;
                            return;
                        }
#pragma unroll
                        for (int i = 0; i < 16; i++)
                            if (col0 + i >= n_valid) sx[i] = 0xFF800000u;
                    }
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        const float s0 = __uint_as_float(sx[i]), s1 = __uint_as_float(sx[i + 1]);
                        float t0, t1;
                        unpack2(fma2(pack2(s0, s1), c2, nm2), t0, t1);
                        float p0, p1;
                        if ((i >> 1) % kH64PolyEvery == kH64PolyEvery - 1) poly_ex2(t0, t1, p0, p1);
                        else p0 = ex2(t0), p1 = ex2(t1);
                        ls2[(i >> 1) & 1] = add2(ls2[(i >> 1) & 1], pack2(p0, p1));
                        p8[i >> 1] = cvt_f16x2(p0, p1);
                    }
                };
                // rolling 16-column chunks: the TMEM load of chunk k+2 runs under the exponentials of chunk k+1
                tmem_ld16(tmem_S + lane_base, sA);
                tmem_ld16(tmem_S + lane_base + 16, sB);
                tmem_wait_ld();
                chunk(sA, preg, 0);
                tmem_ld16(tmem_S + lane_base + 32, sA);
                chunk(sB, preg + 8, 16);
                tmem_wait_ld();
                tmem_ld16(tmem_S + lane_base + 48, sB);
                chunk(sA, preg + 16, 32);
                tmem_wait_ld();
                chunk(sB, preg + 24, 48);
                float l0, l1;
                unpack2(add2(ls2[0], ls2[1]), l0, l1);
                lsum = l0 + l1;
                if (!__any_sync(0xffffffffu, lsum > kRedoSum)) break;
                // O is at rest: the commit behind S[j] covers P[j-1].V[j-1]
                const float m_new = fmaxf(m_ref, step_max(n_valid) * c);
                const float alpha = (m_new == -INFINITY) ? 1.0f : ex2(m_ref - m_new);
                l_run *= alpha;
                if (j > 0) {
#pragma unroll
                    for (int q4 = 0; q4 < HD / 16; q4++) {
                        uint32_t oreg[16];
                        tmem_ld16(tmem_O + lane_base + q4 * 16, oreg);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; i++) oreg[i] = __float_as_uint(__uint_as_float(oreg[i]) * alpha);
                        tmem_st16(tmem_O + lane_base + q4 * 16, oreg);
                    }
                }
                m_ref = m_new;
            }
            l_run += lsum;
            tmem_st32(tmem_P + lane_base, preg);   // over the score columns: this warp has read its lanes of them
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_p_ready);
        }
        if (ok && (!SPLIT || n_tiles > 0)) ok = mbar_wait(bar_o_done, 0, s_abort);
        if constexpr (SPLIT) {
            // O as it is (relative to this CTA's reference), whole rows, chunks swizzled by the row; (m, l) in the Q tile.  The
            // K/V slots and the Q tile are free once the last MMA has completed.
            tc_fence_after();
            float* stage = reinterpret_cast<float*>(smem_gen + kPanelBytes) + r * HD;
            const bool any = ok && n_tiles > 0;
#pragma unroll 1
            for (int q4 = 0; q4 < HD / 16; q4++) {
                uint32_t x[16];
                tmem_ld16(tmem_O + lane_base + q4 * 16, x);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; i += 4)
                    *reinterpret_cast<float4*>(stage + ((((q4 * 16 + i) >> 2) ^ (lane & 7)) << 2)) =
                        any ? make_float4(__uint_as_float(x[i]), __uint_as_float(x[i + 1]), __uint_as_float(x[i + 2]), __uint_as_float(x[i + 3]))
                            : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            reinterpret_cast<float2*>(smem_gen)[r] = make_float2(any ? m_ref : -INFINITY, any ? l_run : 0.0f);
        } else if (ok) {
            tc_fence_after();
            // rows beyond the live ones are written as literal zeros, rows outside the tensor not at all; the K/V slots are
            // free once the last MMA has completed: they stage O
            const float inv = row_live && l_run > 0.0f ? 1.0f / l_run : 0.0f;
            float* stage = reinterpret_cast<float*>(smem_gen + kPanelBytes) + warp * 32 * HD;
#pragma unroll
            for (int q4 = 0; q4 < HD / 32; q4++) {
                uint32_t oreg[32];
                tmem_ld32(tmem_O + lane_base + q4 * 32, oreg);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const float4 o = row_live ? make_float4(__uint_as_float(oreg[i]) * inv, __uint_as_float(oreg[i + 1]) * inv,
                                                            __uint_as_float(oreg[i + 2]) * inv, __uint_as_float(oreg[i + 3]) * inv)
                                              : make_float4(0.f, 0.f, 0.f, 0.f);
                    // OTMA: panels of 32 columns in the copy's own swizzle; else whole rows, chunks swizzled by the row
                    if (OTMA) *reinterpret_cast<float4*>(stage + q4 * 32 * 32 + lane * 32 + (((i >> 2) ^ (lane & 7)) << 2)) = o;
                    else *reinterpret_cast<float4*>(stage + lane * HD + ((((q4 * 32 + i) >> 2) ^ (lane & 7)) << 2)) = o;
                }
            }
            if (OTMA) {
                fence_proxy_async();
                __syncwarp();
                if (lane == 0 && q0 + warp * 32 < rows_total) {
#pragma unroll
                    for (int q4 = 0; q4 < HD / 32; q4++)
                        tma_store_4d(&tmO, smem_u32(stage + q4 * 32 * 32), q4 * 32, hk * a.gqa, (q0 + warp * 32) / a.gqa, b);
                    tma_store_commit_and_wait_read();
                }
            } else {
                float* out = q0 + r < rows_total ? a.dst + (((int64_t)b * a.Tq + iq_dst) * a.dst_heads + h) * HD : nullptr;
                store_o_rows_coalesced<HD>(stage, lane, out);
            }
        }
    }

    if constexpr (SPLIT) {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        // Rows [split * 128 / n_split, ...) of every CTA of the cluster, 16 lanes per row, a float4 each.  All loads of a thread
        // are in flight at once (a loop over the rows paid one round trip of 1 k clk each); peers' memory has been read when
        // this CTA arrives at the second barrier, which it waits for behind its own stores.
        auto merge = [&](auto ns_c) {
            constexpr int NS = decltype(ns_c)::value, ROWS = 16 / NS;   // rows per thread
            const int g4 = tid & 15;
            float w[ROWS][NS], inv[ROWS];
            {
                float2 ml[ROWS][NS];
#pragma unroll
                for (int i = 0; i < ROWS; i++)
#pragma unroll
                    for (int s = 0; s < NS; s++) ml[i][s] = ld_peer_v2(peer_smem(smem_base + (split * (kTile / NS) + i * 8 + (tid >> 4)) * 8, s));
#pragma unroll
                for (int i = 0; i < ROWS; i++) {
                    float M = -INFINITY, L = 0.0f;
#pragma unroll
                    for (int s = 0; s < NS; s++) M = fmaxf(M, ml[i][s].x);
#pragma unroll
                    for (int s = 0; s < NS; s++) {
                        w[i][s] = ml[i][s].x == -INFINITY ? 0.0f : ex2(ml[i][s].x - M);
                        L = fmaf(w[i][s], ml[i][s].y, L);
                    }
                    inv[i] = L > 0.0f ? 1.0f / L : 0.0f;
                }
            }
            float4 x[ROWS][NS];
#pragma unroll
            for (int i = 0; i < ROWS; i++)
#pragma unroll
                for (int s = 0; s < NS; s++) {
                    const int row = split * (kTile / NS) + i * 8 + (tid >> 4);
                    x[i][s] = ld_peer_v4(peer_smem(smem_base + kPanelBytes + (row * HD + ((g4 ^ (row & 7)) << 2)) * 4, s));
                }
#pragma unroll
            for (int i = 0; i < ROWS; i++) {
                const int row = split * (kTile / NS) + i * 8 + (tid >> 4);
                float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int s = 0; s < NS; s++)
                    o.x = fmaf(w[i][s], x[i][s].x, o.x), o.y = fmaf(w[i][s], x[i][s].y, o.y), o.z = fmaf(w[i][s], x[i][s].z, o.z),
                    o.w = fmaf(w[i][s], x[i][s].w, o.w);
                if (q0 + row < rows_total) {
                    const int iq = (q0 + row) / a.gqa, h = hk * a.gqa + (q0 + row) % a.gqa;
                    const bool live = q0 + row < rows_live;
                    reinterpret_cast<float4*>(a.dst + (((int64_t)b * a.Tq + iq) * a.dst_heads + h) * HD)[g4] =
                        live ? make_float4(o.x * inv[i], o.y * inv[i], o.z * inv[i], o.w * inv[i]) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
        };
        if (warp < 4) {
            if (n_split == 2) merge(std::integral_constant<int, 2>{});
            else if (n_split == 4) merge(std::integral_constant<int, 4>{});
            else merge(std::integral_constant<int, 8>{});
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // peers may still read this CTA's rows
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 4) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(128u) : "memory");
    }
}
