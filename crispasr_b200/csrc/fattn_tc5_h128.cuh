// fattn_tc5_h128.cuh — head_dim 128 prefill without an explicit mask, for launches of more than two waves: the kernel of fattn_tc5.cu
// (same roles, tensor memory, stages and arithmetic), whose CTAs take over one another's tiles.
//
// A CTA of a causal launch over a few hundred tokens has one to four key tiles, 1 to 2 us each, in a life of 7 to 13 us: between two CTAs
// on a place of an SM lay 0.8 us, the set-up 1 us, the query tile's copy 1.5 us.  Here a CTA asks the hardware, while its first copies are on
// their way, for a block that has not been launched yet (clusterlaunchcontrol), brings that block's query rows into L2 behind its own
// last copies, and goes on with it: tensor memory and barriers are kept, key tiles and query tiles are counted on for the barriers' phases.
// 8 streams x 407 tokens over a Q8_0 cache 50.9 -> 48.8 us per layer; F16 rows, F32 queries, 16 x 407 68.0 -> 62.9, 2 x 1600 61.8 -> 60.9, 8 x
// 1500 not causal 175.7 -> 170.7; F16 queries, 16 x 407 59.6 -> 56.1, 16 x 750 not causal 103.3 -> 99.7.
// Whoever asks first gets the block, not who is done first: launches of up to two full waves are slower this way (4 x 407 tokens 18.9 ->
// 20.6, 16 x 100 15.5 -> 16.2), so are causal ones of long rows with few tiles more (launch_t), and take the other kernel.  (Asked for behind
// the last copies the answer is waited for: 16 x 750 111.)
// A kernel of its own because the loop around a tile costs the registers that masks need (2 x 1500 under a mask 148 -> 174).

// Asks the hardware for a block of this grid that has not been launched yet and will not be: the caller does its work (16 bytes at `dst`,
// announced on `bar`).  Not again after an answer that there is none.
__device__ __forceinline__ void ask_for_next_block(uint32_t dst, uint32_t bar) {
    mbar_arrive_expect_tx(bar, 16);
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(dst), "r"(bar) : "memory");
}
__device__ __forceinline__ bool next_block(uint32_t src, int& x, int& y, int& z) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b128 r;\n\t"
        "ld.shared.b128 r, [%4];\n\t"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
        "selp.u32 %3, 1, 0, p;\n\t"
        "mov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\t"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%0, %1, %2, _}, r;\n\t}"
        : "=r"(x), "=r"(y), "=r"(z), "=r"(ok)
        : "r"(src)
        : "memory");
    return ok != 0;
}

template <bool RAW>
__global__ void __launch_bounds__(kThreadsTc5, 2)
fattn_prefill_tc5_h128_kernel(const FattnArgs a, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                              const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmO) {
    constexpr int HD = 128, TILE_BYTES = 2 * kPanelBytes;

    extern __shared__ uint8_t smem_dyn[];
    const uint32_t smem_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_dyn + (smem_base - smem_u32(smem_dyn));
    const uint32_t sQ = smem_base, sK = sQ + TILE_BYTES, sV = sK + TILE_BYTES, sBar = sV + TILE_BYTES;
    const uint32_t bar_k_full = sBar, bar_k_empty = sBar + 8, bar_v_full = sBar + 16, bar_v_empty = sBar + 24, bar_s_full = sBar + 32,
                   bar_p_ready = sBar + 40, bar_o_done = sBar + 48, bar_q_full = sBar + 56, bar_q_conv = sBar + 64, bar_next = sBar + 72;
    const uint32_t s_next = sBar + 96;   // the answer about the next block
    uint8_t* misc = smem_gen + 3 * TILE_BYTES + 80;
    // The query tile comes by tensor copies: F16 rows into the operand tile, F32 rows (RAW, 64 KB) as convert_raw_row takes them.
    volatile uint32_t* s_tmem_base = reinterpret_cast<volatile uint32_t*>(misc);
    volatile int* s_abort = reinterpret_cast<volatile int*>(misc + 4);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // tile order and GQA packing as in fattn_prefill_tc5_kernel
    auto place = [&](int x, int y, int z, int& q0, int& hk, int& b) {
        q0 = x * kTile, hk = y, b = z;
        if (a.causal) {
            const int lin = x + gridDim.x * (y + gridDim.y * z), hb = gridDim.y * gridDim.z;
            q0 = (gridDim.x - 1 - lin / hb) * kTile;
            hk = (lin % hb) % gridDim.y, b = (lin % hb) / gridDim.y;
        }
    };
    int q0, hk, b;
    place(blockIdx.x, blockIdx.y, blockIdx.z, q0, hk, b);
    auto prefetch_q = [&](int q0, int hk, int b) {
        constexpr int kCols = RAW ? 32 : 64;
#pragma unroll
        for (int p = 0; p < HD / kCols; p++) tma_prefetch_4d(&tmQ, p * kCols, hk * a.gqa, q0 / a.gqa, b);
    };
    if (tid == 4 * 32) prefetch_q(q0, hk, b);
    // launched with programmatic stream serialisation: but for that, nothing is read or written before the previous kernel of the stream
    // has completed and flushed
    wait_for_predecessors();
    // ---- set-up ----
    if (tid == 4 * 32) {
        for (int i = 0; i < 10; i++) {
            const uint32_t bar = sBar + 8 * i;
            mbar_init(bar, bar == bar_p_ready || bar == bar_q_conv ? 4 : 1);   // four: one arrival per softmax warp
        }
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmK)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmV)) : "memory");
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(const_cast<uint32_t*>(s_tmem_base))),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // One query tile; `base` key tiles and `item` query tiles with keys came before it in this CTA (the phases of the barriers), `turn`
    // counts all of them.  Returns its key tiles.
    auto run_tile = [&](int q0, int hk, int b, uint32_t base, uint32_t item, uint32_t turn) -> int {
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
            if (tid == 4 * 32) ask_for_next_block(s_next, bar_next);
            if (turn == 0) __syncthreads();   // a first tile without keys: nobody else has seen the set-up of the barriers yet
            return 0;
        }
        auto load_kv = [&](const CUtensorMap& tm, uint32_t stage, uint32_t bar, int j) {
            mbar_arrive_expect_tx(bar, TILE_BYTES);
            tma_load_4d(stage, &tm, bar, 0, j * kTile, hk, bk);
            tma_load_4d(stage + kPanelBytes, &tm, bar, 64, j * kTile, hk, bk);
        };
        if (tid == 4 * 32) {
            mbar_arrive_expect_tx(bar_q_full, RAW ? 2 * TILE_BYTES : TILE_BYTES);
            if (RAW) {
#pragma unroll
                for (int p = 0; p < 4; p++) tma_load_4d(sQ + raw_panel_off(p), &tmQ, bar_q_full, p * 32, hk * a.gqa, q0 / a.gqa, b);
            } else {
#pragma unroll
                for (int p = 0; p < 2; p++) tma_load_4d(sQ + p * kPanelBytes, &tmQ, bar_q_full, p * 64, hk * a.gqa, q0 / a.gqa, b);
            }
            load_kv(tmK, sK, bar_k_full, 0);
            if (!RAW) load_kv(tmV, sV, bar_v_full, 0);   // (the V stage holds raw query rows for now)
            ask_for_next_block(s_next, bar_next);
        }
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        const uint32_t tmem_base = __shfl_sync(0xffffffffu, *s_tmem_base, 0);
        const uint32_t tmem_S = tmem_base, tmem_P = tmem_base, tmem_O = tmem_base + kTile;   // P as f16x2 over the first 64 columns of S
        if constexpr (RAW) {
            if (warp < 4) {
                const bool there = mbar_wait(bar_q_full, item & 1, s_abort);
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
                int issued_k = 1, issued_v = RAW ? 0 : 1;
                if (RAW) {
                    ok = mbar_wait(bar_q_conv, item & 1, s_abort);
                    if (ok) load_kv(tmV, sV, bar_v_full, 0), issued_v = 1;
                }
                for (int j = 1; j < n_tiles && ok; j++) {
                    ok = mbar_wait(bar_k_empty, (base + j - 1) & 1, s_abort);
                    if (!ok) break;
                    load_kv(tmK, sK, bar_k_full, j);
                    issued_k = j + 1;
                    ok = mbar_wait(bar_v_empty, (base + j - 1) & 1, s_abort);
                    if (!ok) break;
                    load_kv(tmV, sV, bar_v_full, j);
                    issued_v = j + 1;
                }
                if (ok) {   // the query rows of the next tile into L2, behind the last copies of this one
                    int x, y, z, nq0, nhk, nb;
                    if (mbar_wait(bar_next, turn & 1, s_abort) && next_block(s_next, x, y, z)) {
                        place(x, y, z, nq0, nhk, nb);
                        prefetch_q(nq0, nhk, nb);
                    }
                }
                if (!ok) {
                    // drain: wait (bounded) for the copies this thread still has in flight
                    for (uint32_t it = 0; it < 4096 && !mbar_try_wait(bar_q_full, item & 1); ++it) __nanosleep(256);
                    for (uint32_t it = 0; it < 4096 && !mbar_try_wait(bar_k_full, (base + issued_k - 1) & 1); ++it) __nanosleep(256);
                    for (uint32_t it = 0; it < 4096 && issued_v > 0 && !mbar_try_wait(bar_v_full, (base + issued_v - 1) & 1); ++it) __nanosleep(256);
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
                auto issue_s = [&]() {
                    issue_scores<HD>(tmem_S, q_lo, k_lo);
                    tc_commit(bar_s_full);
                    tc_commit(bar_k_empty);
                };
                bool ok = mbar_wait(bar_k_full, base & 1, s_abort) && mbar_wait(RAW ? bar_q_conv : bar_q_full, item & 1, s_abort);
                ok = warp_all(ok);
                if (ok) {
                    tc_fence_after();
                    if (elect_one()) issue_s();
                    __syncwarp();
                }
                for (int j = 0; j < n_tiles && ok; j++) {
                    const bool more = j + 1 < n_tiles;
                    ok = mbar_wait(bar_v_full, (base + j) & 1, s_abort);
                    if (ok && more) ok = mbar_wait(bar_k_full, (base + j + 1) & 1, s_abort);
                    if (ok) ok = mbar_wait(bar_p_ready, (base + j) & 1, s_abort);
                    ok = warp_all(ok);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        issue_pv<HD>(tmem_O, tmem_P, v_lo, j == 0);
                        tc_commit(bar_v_empty);
                        if (more) issue_s();
                        if (!more) tc_commit(bar_o_done);
                    }
                    __syncwarp();
                }
                if (!ok) {
                    // make sure no MMA of this CTA is still running before TMEM is released (the commit comes from the lane that
                    // issued them)
                    if (elect_one()) tc_commit(bar_o_done);
                    __syncwarp();
                    for (uint32_t it = 0; it < 65536 && !mbar_try_wait(bar_o_done, item & 1); ++it) __nanosleep(256);
                }
                __syncwarp();
            }
        } else {
            // ================= softmax / correction / epilogue =================
            const int r = tid;
            const bool row_live = q0 + r < rows_live;
            const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
            const float c = a.scale * kLog2e;
            int kend = len_b;
            if (a.causal) kend = min(kend, n_past + (row_live ? (q0 + r) / a.gqa : a.Tq) + 1);
            float m_ref = -INFINITY, l_run = 0.0f;
            bool ok = true;
            for (int j = 0; j < n_tiles; j++) {
                ok = mbar_wait(bar_s_full, (base + j) & 1, s_abort);
                if (!ok) break;
                tc_fence_after();
                const int n_valid = kend - j * kTile;  // columns >= n_valid of this row are masked
                const bool full_tile = __all_sync(0xffffffffu, n_valid >= kTile);
                if (j == 0) m_ref = first_maximum(tmem_S + lane_base, n_valid) * c;
                uint32_t preg[2][32];
                float lsum = 0.0f;
                for (int attempt = 0; attempt < 2; attempt++) {
                    // P = exp2(S*c - m_ref), rounded to f16x2; the tile maximum is tracked in the same pass and
                    // only checked afterwards (lazy rescale).
                    const float m_use = (m_ref == -INFINITY) ? 0.0f : m_ref;
                    float mx;
                    softmax_tile(tmem_S + lane_base, c, m_use, full_tile, n_valid, preg, mx, lsum, []() {});
                    const float m_tile = c * mx;
                    const bool grow = m_tile > m_ref + kRescaleThreshold;
                    if (!__any_sync(0xffffffffu, grow)) break;
                    // some row of this warp outgrew its reference maximum: rescale O and l, then redo P
                    // (O is at rest: the commit behind S[j] covers P[j-1].V[j-1])
                    const float m_new = fmaxf(m_ref, m_tile);
                    const float alpha = (m_new == -INFINITY) ? 1.0f : ex2(m_ref - m_new);
                    l_run *= alpha;
                    if (j > 0) rescale_o<HD>(tmem_O + lane_base, alpha);
                    m_ref = m_new;
                }
                l_run += lsum;
                tmem_st32(tmem_P + lane_base, preg[0]);
                tmem_st32(tmem_P + lane_base + 32, preg[1]);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_p_ready);
            }
            if (ok) ok = mbar_wait(bar_o_done, item & 1, s_abort);
            if (ok) {
                tc_fence_after();
                // dead rows are written as literal zeros, rows outside the tensor not at all; the K and V stages are free once the last MMA has
                // completed: they stage O
                const float inv = row_live && l_run > 0.0f ? 1.0f / l_run : 0.0f;
                float* stage = reinterpret_cast<float*>(smem_gen + TILE_BYTES) + warp * 32 * HD;
                store_o_box<HD>(tmO, stage, tmem_O + lane_base, inv, row_live, lane, q0 + warp * 32, rows_total, hk, a.gqa, b);
            }
        }
        return n_tiles;
    };
    uint32_t base = 0, item = 0;
    for (uint32_t turn = 0;; turn++) {
        const int n = run_tile(q0, hk, b, base, item, turn);
        // the stages, the tensor memory and the answer's place are free for the next tile behind this
        int x, y, z;
        const bool more = mbar_wait(bar_next, turn & 1, s_abort) && next_block(s_next, x, y, z);
        fence_proxy_async();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (!more || *s_abort) break;
        base += n, item += n > 0;
        place(x, y, z, q0, hk, b);
    }

    // ---- teardown ----
    if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*s_tmem_base), "r"(kTmemCols) : "memory");
}

