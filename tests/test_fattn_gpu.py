"""Parity of the CUDA operator (through the C-ABI) against the CPU oracle on seeded inputs.
Tolerance: max-abs <= 2e-3 and relative L2 <= 1e-3 (fp32 softmax, fp32 accumulation)."""
import os

import numpy as np
import pytest
import torch

from crispasr_b200 import abi
from tests.util import assert_close, cuda_view, errors, gpu_op, randn_f16

pytestmark = pytest.mark.gpu
G = os.path.join(os.path.dirname(__file__), "golden")

KERNELS = {"auto": abi.KERNEL_NONE, "tile": abi.KERNEL_TILE_MMA}


@pytest.fixture(params=list(KERNELS))
def kernel(request, b200):
    """Runs each case with the automatic kernel choice and again forced onto the general tile kernel."""
    b200.lib().b200_set_kernel_override(KERNELS[request.param])
    yield request.param
    b200.lib().b200_set_kernel_override(abi.KERNEL_NONE)


def test_extension_is_loaded_and_device_is_b200(b200):
    assert torch.cuda.is_available()
    assert torch.cuda.get_device_capability(0)[0] == 10
    assert os.path.exists(b200.LIB_PATH)
    # the library under test was linked from the sources now in the tree (stamp written at link time)
    from crispasr_b200 import build
    assert build.built_hash() == build.source_hash()
    loaded = [ln.split()[-1] for ln in open("/proc/self/maps") if "libb200_fattn.so" in ln]
    assert loaded and os.path.realpath(loaded[0]) == os.path.realpath(b200.LIB_PATH)


def test_bounded_wait_runs_out_sets_status_and_leaves_the_context_usable(b200, orc):
    """Failure path of the device-side waits, without a fault: a one-warp probe kernel waits on an mbarrier that
    nothing completes, gives up after a few thousand polls, sets the status word and returns.  The host then reads
    B200_E_DEVICE_WAIT, clears it, and the next ordinary launch is green."""
    L = b200.lib()
    assert L.b200_device_status_reset() == 0 and L.b200_device_status() == 0
    assert L.b200_test_bounded_wait(0, None) == abi.E_LIMIT
    assert L.b200_test_bounded_wait(4096, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert L.b200_device_status() == abi.E_DEVICE_WAIT
    assert L.b200_device_status() == abi.E_DEVICE_WAIT, "the word is sticky until it is reset"
    assert L.b200_device_status_reset() == 0 and L.b200_device_status() == 0
    rng = np.random.default_rng(3)
    q, k, v = (randn_f16(rng, (1, 4, 200, 64)) for _ in range(3))
    assert_close(gpu_op(b200, q, k, v, scale=0.125), orc.flash_attn_ext(q, k, v, scale=0.125), "launch after a run-out wait")
    kq = orc.quantize_q8_0(rng.standard_normal((2, 2, 300, 128)).astype(np.float32))
    qd = randn_f16(rng, (2, 8, 1, 128))
    assert_close(gpu_op(b200, qd, kq, kq, scale=128 ** -0.5, kv_type=abi.Q8_0),
                 orc.flash_attn_ext(qd, kq, kq, scale=128 ** -0.5, kv_type=abi.Q8_0), "Q8_0 decode after a run-out wait")
    assert L.b200_device_status() == 0


# ---- config 1: Whisper base.en encoder self-attention --------------------------------------------
def test_cfg1_whisper_base_encoder(b200, orc, kernel):
    rng = np.random.default_rng(0)
    T, H, hd = 1500, 8, 64
    q, k, v = (randn_f16(rng, (1, H, T, hd)) for _ in range(3))
    ref = orc.flash_attn_ext(q, k, v, scale=0.125)
    got = gpu_op(b200, q.astype(np.float32), k, v, scale=0.125)   # Q is F32 at the reference call site
    assert_close(got, ref, "cfg1 contiguous, F32 Q")
    assert_close(gpu_op(b200, q, k, v, scale=0.125), ref, "cfg1 contiguous, F16 Q")


def test_cfg1_whisper_strided_padded_views(b200, orc, kernel):
    """What src/crispasr.cpp:2813-2821 really issues: token-major K/V views (nb1 = 2*n_state, nb2 = 2*hd)
    over a zero-cleared buffer padded to 1536 rows, no mask: the 36 zero rows take part in the softmax."""
    rng = np.random.default_rng(0)
    T, Tp, H, hd = 1500, 1536, 8, 64
    kbuf = np.zeros((1, Tp, H, hd), np.float16)
    vbuf = np.zeros((1, Tp, H, hd), np.float16)
    kbuf[:, :T], vbuf[:, :T] = randn_f16(rng, (1, T, H, hd)), randn_f16(rng, (1, T, H, hd))
    qbuf = randn_f16(rng, (1, T, H, hd)).astype(np.float32)
    qv, kv, vv = (x.transpose(0, 2, 1, 3) for x in (qbuf, kbuf, vbuf))     # (B,H,T,hd) strided
    ref = orc.flash_attn_ext(qv, kv, vv, scale=0.125)
    got = gpu_op(b200, cuda_view(qv, qbuf), cuda_view(kv, kbuf), cuda_view(vv, vbuf), scale=0.125)
    assert_close(got, ref, "cfg1 whisper-strided, Lk 1536 with 36 zero rows")


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("gqa", [1, 2, 4])
@pytest.mark.parametrize("form", ["plain", "causal", "q_len", "mask"])
@pytest.mark.parametrize("q_f32", [False, True])
def test_prefill_query_views(b200, orc, hd, gqa, form, q_f32):
    """Query rows take the tensor-copy path in and out of the tcgen05 kernel, as boxes of [columns, heads of the
    group, tokens] (F16 straight into the operand tile; F32 at head_dim 128 raw into the K and V stages and converted
    from there, at head_dim 64 through registers): token-major strided Q views (nb1 = H * hd * elements), one to four heads per KV head, two batch entries,
    a last query tile that ends inside the box (Q rows beyond Tq read as zeros, output rows beyond Tq are clipped),
    ragged q_len (rows at or beyond it are written as zeros), the causal tile order, an explicit mask."""
    rng = np.random.default_rng(4100 + hd + gqa)
    B, T, H = 2, 300, 4
    Hkv = H // gqa
    qbuf = randn_f16(rng, (B, T, H, hd))
    if q_f32:
        qbuf = qbuf.astype(np.float32)
    kbuf, vbuf = randn_f16(rng, (B, T, Hkv, hd)), randn_f16(rng, (B, T, Hkv, hd))
    qv, kv, vv = (x.transpose(0, 2, 1, 3) for x in (qbuf, kbuf, vbuf))     # (B, H, T, hd) strided
    kw = dict(scale=hd ** -0.5)
    mask = None
    if form == "causal":
        kw.update(causal=True, n_past=0)
        mask_ref = np.triu(np.full((T, T), -np.inf, np.float32), 1).astype(np.float16)[None, None]
        ref = orc.flash_attn_ext(qv, kv, vv, mask_ref, scale=kw["scale"])
    elif form == "q_len":
        kw.update(q_len=[T, 130], kv_len=[T, 130])
        ref = orc.flash_attn_ext(qv, kv, vv, scale=kw["scale"], kv_len=[T, 130])
        ref[1, 130:] = 0.0   # (B, Tq, H, hd)
    else:
        if form == "mask":
            mask = np.where(rng.random((1, 1, T, T)) < 0.3, -np.inf, 0.0).astype(np.float16)
            mask[..., 0] = 0
        ref = orc.flash_attn_ext(qv, kv, vv, mask, **kw)
    got = gpu_op(b200, cuda_view(qv, qbuf), cuda_view(kv, kbuf), cuda_view(vv, vbuf), mask, **kw)
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5
    if form == "q_len":
        assert not got[1, 130:].any(), "rows at or beyond q_len must be zeros"
    assert_close(got, ref, f"strided Q views hd={hd} gqa={gqa} {form} f32={q_f32}")


# ---- config 2: Whisper large-v3 decoder step, beam 5 ------------------------------------------------
@pytest.mark.parametrize("L", [1, 64, 224, 448])
def test_cfg2_decoder_self_attention_beam_cells(b200, orc, kernel, L):
    """Layout A of the reference: one pooled cell cache shared by 5 beams, membership only in the F16
    mask [n_kv, 5] built by the rule of src/crispasr.cpp:3480-3488; Q and K pre-scaled, scale 1.0."""
    rng = np.random.default_rng(1)
    H, hd, beams = 20, 64, 5
    shared = L // 2                      # shared prompt prefix, then private suffixes
    priv = L - shared
    n_cells = shared + beams * priv
    n_kv = min(3584, max(256, -(-n_cells // 256) * 256))
    cell_pos = np.full(n_kv, 10 ** 6, np.int32)      # unused cells: never visible
    bits = np.zeros(n_kv, np.uint32)
    cell_pos[:shared], bits[:shared] = np.arange(shared), (1 << beams) - 1
    for j in range(beams):
        sl = slice(shared + j * priv, shared + (j + 1) * priv)
        cell_pos[sl], bits[sl] = shared + np.arange(priv), 1 << j
    mask = orc.whisper_beam_mask(cell_pos, bits, tok_seq=np.arange(beams), tok_pos=np.full(beams, L - 1))
    mask = mask[None, None]                                   # (1,1,5,n_kv)
    kbuf = randn_f16(rng, (1, n_kv, H, hd), 0.5)
    vbuf = randn_f16(rng, (1, n_kv, H, hd), 0.5)
    q = randn_f16(rng, (1, H, beams, hd), 0.5).astype(np.float32)
    kv, vv = kbuf.transpose(0, 2, 1, 3), vbuf.transpose(0, 2, 1, 3)
    ref = orc.flash_attn_ext(q, kv, vv, mask, scale=1.0)
    got = gpu_op(b200, q, cuda_view(kv, kbuf), cuda_view(vv, vbuf), mask, scale=1.0)
    assert_close(got, ref, f"cfg2 self L={L}")


@pytest.mark.parametrize("segments,Lk", [(1, 1500), (1, 1536), (3, 1500)])
def test_cfg2_decoder_cross_attention(b200, orc, kernel, segments, Lk):
    rng = np.random.default_rng(1)
    H, hd, beams = 20, 64, 5
    kbuf = np.zeros((segments, 1536, H, hd), np.float16)
    vbuf = np.zeros_like(kbuf)
    kbuf[:, :1500], vbuf[:, :1500] = randn_f16(rng, (segments, 1500, H, hd), 0.5), randn_f16(rng, (segments, 1500, H, hd), 0.5)
    q = randn_f16(rng, (segments, H, beams, hd), 0.5).astype(np.float32)
    kv, vv = kbuf.transpose(0, 2, 1, 3)[:, :, :Lk], vbuf.transpose(0, 2, 1, 3)[:, :, :Lk]
    scale = 64 ** -0.25
    ref = orc.flash_attn_ext(q, kv, vv, scale=scale)
    got = gpu_op(b200, q, cuda_view(kv, kbuf), cuda_view(vv, vbuf), scale=scale)
    assert_close(got, ref, f"cfg2 cross segments={segments} Lk={Lk}")
    if kernel == "auto":
        assert b200.lib().b200_last_kernel() == abi.KERNEL_DECODE_SPLIT


# ---- config 3: Whisper large-v3 encoder prefill ---------------------------------------------------------
def test_cfg3_large_v3_encoder_segments(b200, orc, kernel):
    rng = np.random.default_rng(2)
    S, H, T, hd = 2, 20, 1500, 64
    q, k, v = (randn_f16(rng, (S, H, T, hd)) for _ in range(3))
    ref = orc.flash_attn_ext(q, k, v, scale=0.125)
    assert_close(gpu_op(b200, q, k, v, scale=0.125), ref, "cfg3 two segments")
    if kernel == "auto":
        assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5, "the encoder prefill must run on the tcgen05 kernel"
        assert b200.lib().b200_device_status() == 0


@pytest.mark.parametrize("env", ["B200_HOST_CHUNKS=1", "B200_HOST_CHUNKS=16", "B200_DECODE_CLUSTER_MERGE=0", "B200_DECODE_CTAS_PER_SM=1"])
def test_switches_read_once_per_process(env):
    """Each of the library's environment variables is read once per process: decode steps that split their keys and
    host-buffer calls run against the oracle in a child process that has it set."""
    import subprocess
    import sys

    name, value = env.split("=")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, os.path.join(root, "tests", "variant_case.py")], env={**os.environ, name: value},
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert r.stdout.count("OK") == 4, r.stdout


def test_voxtral_audio_encoder_f32_kv(b200, orc, kernel):
    """core_attn::encoder_self_attn (src/core/attention.h:517-580): contiguous F32 Q/K/V, Whisper large dims, no pad,
    no mask.  K/V are converted to F16 by a pre-pass into the workspace and the call runs on the tcgen05 kernel."""
    rng = np.random.default_rng(22)
    H, T, hd = 20, 1500, 64
    q, k, v = (randn_f16(rng, (1, H, T, hd)).astype(np.float32) for _ in range(3))
    ref = orc.flash_attn_ext(q, k, v, scale=0.125)
    assert_close(gpu_op(b200, q, k, v, scale=0.125), ref, "voxtral encoder, F32 K/V")
    if kernel == "auto":
        assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5
        assert b200.workspace_bytes(torch.from_numpy(q), torch.from_numpy(k), torch.from_numpy(v), scale=0.125) >= 2 * H * T * hd * 2


@pytest.mark.parametrize("hd,per_head", [(64, False), (128, True)])
def test_explicit_mask_prefill(b200, orc, kernel, hd, per_head):
    """Explicit F16 masks with 16-byte aligned rows (LLM causal prefill mask of src/voxtral.cpp:1187-1194 plus random
    additive bias and -inf holes, shared or per head) on the tcgen05 kernel."""
    rng = np.random.default_rng(hd)
    B, H, Hkv, Tq, Lk = 2, 4, 2, 300, 520
    q, k, v = randn_f16(rng, (B, H, Tq, hd)), randn_f16(rng, (B, Hkv, Lk, hd)), randn_f16(rng, (B, Hkv, Lk, hd))
    m = (rng.standard_normal((1, H if per_head else 1, Tq, Lk)) * 0.5).astype(np.float16)
    m[rng.random(m.shape) < 0.3] = -np.inf
    m[..., 0] = 0
    m = m + orc.causal_mask(Lk, Tq, Lk - Tq)[None, None]
    m[0, 0, 17, :] = -np.inf                      # one fully masked row
    ref = orc.flash_attn_ext(q, k, v, m, scale=hd ** -0.5)
    got = gpu_op(b200, q, k, v, m, scale=hd ** -0.5)
    assert np.all(got[:, 17, 0] == 0)
    assert_close(got, ref, f"explicit mask hd={hd} per_head={per_head}")
    if kernel == "auto":
        assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5


# ---- config 4: Voxtral-style LLM decoder, GQA 32/8, hd 128, Q8_0 KV ------------------------------------------
def _q8_cache(orc, rng, streams, Hkv, rows, hd, max_ctx):
    x = rng.standard_normal((streams, Hkv, rows, hd)).astype(np.float32)
    cache = np.zeros((streams, Hkv, max_ctx, hd // 32 * 34), np.uint8)
    cache[:, :, :rows] = orc.quantize_q8_0(x)
    return cache


def test_cfg4_prefill_causal_q8_0(b200, orc, kernel):
    rng = np.random.default_rng(3)
    T, H, Hkv, hd = 407, 32, 8, 128
    kc, vc = _q8_cache(orc, rng, 1, Hkv, T, hd, 448), _q8_cache(orc, rng, 1, Hkv, T, hd, 448)
    q = randn_f16(rng, (1, H, T, hd)).astype(np.float32)
    scale = hd ** -0.5
    kv, vv = kc[:, :, :T], vc[:, :, :T]
    mask = orc.causal_mask(T, T, 0)[None, None]
    ref = orc.flash_attn_ext(q, kv, vv, mask, scale=scale, kv_type=abi.Q8_0)
    got_m = gpu_op(b200, q, cuda_view(kv, kc), cuda_view(vv, vc), mask, scale=scale, kv_type=abi.Q8_0)
    assert_close(got_m, ref, "cfg4 prefill, explicit F16 causal mask")
    got_i = gpu_op(b200, q, cuda_view(kv, kc), cuda_view(vv, vc), scale=scale, kv_type=abi.Q8_0, causal=True, n_past=0)
    assert_close(got_i, ref, "cfg4 prefill, implicit causal")


@pytest.mark.parametrize("lens", [[408] * 8, [408, 450, 511, 512, 513, 600, 663, 1]])
def test_cfg4_decode_ragged_streams(b200, orc, kernel, lens):
    rng = np.random.default_rng(3)
    S, H, Hkv, hd, max_ctx = 8, 32, 8, 128, 672
    kc, vc = _q8_cache(orc, rng, S, Hkv, max_ctx, hd, max_ctx), _q8_cache(orc, rng, S, Hkv, max_ctx, hd, max_ctx)
    q = randn_f16(rng, (S, H, 1, hd)).astype(np.float32)
    scale = hd ** -0.5
    Lk = max(lens)
    kv, vv = kc[:, :, :Lk], vc[:, :, :Lk]
    ref = orc.flash_attn_ext(q, kv, vv, scale=scale, kv_type=abi.Q8_0, kv_len=lens)
    got = gpu_op(b200, q, cuda_view(kv, kc), cuda_view(vv, vc), scale=scale, kv_type=abi.Q8_0, kv_len=lens)
    assert_close(got, ref, f"cfg4 decode lens={lens}")
    if kernel == "auto":
        assert b200.lib().b200_last_kernel() == abi.KERNEL_DECODE_SPLIT


@pytest.mark.parametrize("hd", [32, 64, 128])
@pytest.mark.parametrize("form", ["plain", "causal3", "mask", "softcap"])
def test_q8_0_decode_forms(b200, orc, kernel, hd, form):
    """Q8_0 cache decode at every head dim with its own staging form (32: staged dequantise, 64 / 128: register
    dequantise) through the general softmax path: multi-token causal decode, explicit mask, softcap, ragged lengths."""
    rng = np.random.default_rng(100 + hd)
    S, H, Hkv, max_ctx = 3, 8, 2, 352
    lens = [333, 64, 201]
    Tq = 3 if form == "causal3" else 1
    kc, vc = _q8_cache(orc, rng, S, Hkv, max_ctx, hd, max_ctx), _q8_cache(orc, rng, S, Hkv, max_ctx, hd, max_ctx)
    q = randn_f16(rng, (S, H, Tq, hd)).astype(np.float32)
    Lk = max(lens)
    kv, vv = kc[:, :, :Lk], vc[:, :, :Lk]
    kw = dict(scale=hd ** -0.5, kv_type=abi.Q8_0)
    mask = None
    if form == "causal3":
        # three new tokens at the end of each stream: row i sees keys < len - 2 + i; expressed as explicit masks for the oracle
        mask = np.zeros((S, 1, Tq, Lk), np.float16)
        for b, n in enumerate(lens):
            for i in range(Tq):
                mask[b, 0, i, n - (Tq - 1) + i:] = -np.inf
        ref = orc.flash_attn_ext(q, kv, vv, mask, **kw)
        got = np.stack([gpu_op(b200, q[b:b + 1], cuda_view(kv[b:b + 1, :, :lens[b]], kc), cuda_view(vv[b:b + 1, :, :lens[b]], vc),
                               causal=True, n_past=lens[b] - Tq, **kw)[0] for b in range(S)])
    else:
        if form == "mask":
            mask = np.where(rng.random((S, 1, Tq, Lk)) < 0.3, -np.inf, 0.0).astype(np.float16)
            mask[..., 0] = 0
        if form == "softcap":
            kw["softcap"] = 5.0
        ref = orc.flash_attn_ext(q, kv, vv, mask, kv_len=lens, **kw)
        got = gpu_op(b200, q, cuda_view(kv, kc), cuda_view(vv, vc), mask, kv_len=lens, **kw)
    assert_close(got, ref, f"Q8_0 decode hd={hd} {form}")
    if kernel == "auto":
        assert b200.lib().b200_last_kernel() == abi.KERNEL_DECODE_SPLIT


@pytest.mark.parametrize("n_splits", [1, 2, 3, 5, 8, 9, 64])
@pytest.mark.parametrize("kv_kind", ["q8_0", "f16"])
def test_decode_forced_split_counts(b200, orc, n_splits, kv_kind):
    """Every way the partial results of the KV splits are merged: none (one split), inside a thread-block cluster
    (Q8_0 cache, 2..8 splits), through the workspace and the merge kernel (the rest); ragged lengths leave some
    splits without a key."""
    rng = np.random.default_rng(700 + n_splits)
    S, H, Hkv, hd, max_ctx = 3, 8, 2, 128, 640
    lens = [600, 65, 330]
    q = randn_f16(rng, (S, H, 1, hd)).astype(np.float32)
    kw = dict(scale=hd ** -0.5, kv_len=lens)
    if kv_kind == "q8_0":
        kc, vc = _q8_cache(orc, rng, S, Hkv, max_ctx, hd, max_ctx), _q8_cache(orc, rng, S, Hkv, max_ctx, hd, max_ctx)
        kw["kv_type"] = abi.Q8_0
    else:
        kc, vc = randn_f16(rng, (S, Hkv, max_ctx, hd)), randn_f16(rng, (S, Hkv, max_ctx, hd))
    kv, vv = kc[:, :, :600], vc[:, :, :600]
    ref = orc.flash_attn_ext(q, kv, vv, **kw)
    assert b200.lib().b200_set_decode_splits(n_splits) == 0
    try:
        tq, tk, tv = (torch.from_numpy(np.ascontiguousarray(x)) for x in (q, kv, vv))
        assert b200.plan(tq, tk, tv, **{k: v for k, v in kw.items() if k != "kv_len"})[1] == min(n_splits, 10)
        got = gpu_op(b200, q, cuda_view(kv, kc), cuda_view(vv, vc), **kw)
    finally:
        assert b200.lib().b200_set_decode_splits(0) == 0
    assert_close(got, ref, f"decode {kv_kind}, {n_splits} splits forced")


@pytest.mark.parametrize("n_splits", [2, 5, 8])
@pytest.mark.parametrize("shape", [("f16", 64, 5, 1, False), ("f16", 64, 5, 1, True), ("f16", 64, 3, 4, False), ("f16", 128, 4, 4, False),
                                   ("q8_0", 128, 4, 4, False), ("q8_0", 64, 2, 4, False), ("q8_0", 128, 3, 4, True)])
def test_cluster_merge_row_counts(b200, orc, n_splits, shape):
    """The merge inside a thread-block cluster with 5, 8, 12 and 16 query rows per KV head (the receive area of a CTA
    is sized by the row count), head dims 64 and 128, both cache types, with and without an explicit mask; ragged
    lengths leave some CTAs of a cluster without a key."""
    kv_kind, hd, Tq, gqa, masked = shape
    rng = np.random.default_rng(900 + n_splits + hd + Tq)
    S, Hkv, max_ctx, Lk = 2, 2, 704, 640
    H = Hkv * gqa
    lens = [640, 130]
    q = randn_f16(rng, (S, H, Tq, hd)).astype(np.float32)
    kw = dict(scale=hd ** -0.5, kv_len=lens)
    if kv_kind == "q8_0":
        kc, vc = _q8_cache(orc, rng, S, Hkv, max_ctx, hd, max_ctx), _q8_cache(orc, rng, S, Hkv, max_ctx, hd, max_ctx)
        kw["kv_type"] = abi.Q8_0
    else:
        kc, vc = randn_f16(rng, (S, Hkv, max_ctx, hd)), randn_f16(rng, (S, Hkv, max_ctx, hd))
    kv, vv = kc[:, :, :Lk], vc[:, :, :Lk]
    mask = None
    if masked:
        mask = np.where(rng.random((S, 1, Tq, Lk)) < 0.3, -np.inf, 0.0).astype(np.float16)
        mask[..., 0] = 0
    ref = orc.flash_attn_ext(q, kv, vv, mask, **kw)
    assert b200.lib().b200_set_decode_splits(n_splits) == 0
    try:
        got = gpu_op(b200, q, cuda_view(kv, kc), cuda_view(vv, vc), mask, **kw)
        assert b200.lib().b200_last_kernel() == abi.KERNEL_DECODE_SPLIT
    finally:
        assert b200.lib().b200_set_decode_splits(0) == 0
    assert_close(got, ref, f"cluster merge {kv_kind} hd={hd} rows={Tq * gqa} mask={masked}, {n_splits} splits")


def test_cfg4_decode_f16_cache_gqa(b200, orc, kernel):
    rng = np.random.default_rng(33)
    S, H, Hkv, hd, Lk = 4, 32, 8, 128, 535
    k, v = randn_f16(rng, (S, Hkv, Lk, hd)), randn_f16(rng, (S, Hkv, Lk, hd))
    q = randn_f16(rng, (S, H, 1, hd)).astype(np.float32)
    ref = orc.flash_attn_ext(q, k, v, scale=hd ** -0.5)
    assert_close(gpu_op(b200, q, k, v, scale=hd ** -0.5), ref, "decode F16 GQA")


# ---- config 5: FastConformer relative-position attention ---------------------------------------------------------
def _relpos_case(orc, rng, T, H=8, hd=128, d_model=1024):
    q = rng.standard_normal((1, H, T, hd)).astype(np.float32)
    u = (rng.standard_normal((H, 1, hd)) * 0.02).astype(np.float32)
    vb = (rng.standard_normal((H, 1, hd)) * 0.02).astype(np.float32)
    q_u = (q + u).astype(np.float16).astype(np.float32)
    q_v = (q + vb).astype(np.float16).astype(np.float32)
    k, v = randn_f16(rng, (1, H, T, hd)).astype(np.float32), randn_f16(rng, (1, H, T, hd)).astype(np.float32)
    pe = orc.make_pos_enc(d_model, T)                                        # (2T-1, d)
    w = (rng.standard_normal((d_model, H * hd)) / 32.0).astype(np.float32)   # attn_pos_w, sigma 1/32
    r = (pe @ w).reshape(2 * T - 1, H, hd).transpose(1, 0, 2)[None]
    r = np.ascontiguousarray(r).astype(np.float16)
    return q_u, q_v, k, v, r


@pytest.mark.parametrize("T", [64, 200, 611])
def test_cfg5_fused_relpos_bias(b200, orc, kernel, T):
    """Fused bias == the reference's materialised F16 mask path (src/core/fastconformer.h:880-933)."""
    rng = np.random.default_rng(4)
    q_u, q_v, k, v, r = _relpos_case(orc, rng, T)
    scale = 128 ** -0.5
    mask = orc.relpos_mask(q_v, r, scale)                       # (1,H,T,T) F16: what the reference feeds the op
    ref = orc.flash_attn_ext(q_u, k, v, mask, scale=scale)
    got_fused = gpu_op(b200, q_u, k, v, scale=scale, q_v=q_v, r=r)
    assert_close(got_fused, ref, f"cfg5 fused T={T}")
    got_f32r = gpu_op(b200, q_u, k, v, scale=scale, q_v=q_v, r=r.astype(np.float32))   # R as the runtimes hold it (F32)
    assert_close(got_f32r, ref, f"cfg5 fused, F32 R, T={T}")
    got_mask = gpu_op(b200, q_u, k, v, mask, scale=scale)       # per-head mask form of the plain op
    assert_close(got_mask, ref, f"cfg5 per-head mask T={T}")


def test_cfg5_relpos_with_padding_mask(b200, orc, kernel):
    """Bucketed padding (src/canary_ctc.cpp:370-382): pad keys carry -inf on top of the bias."""
    rng = np.random.default_rng(44)
    T, valid = 160, 131
    q_u, q_v, k, v, r = _relpos_case(orc, rng, T)
    scale = 128 ** -0.5
    pad = np.zeros((1, 1, T, T), np.float16)
    pad[..., valid:] = -np.inf
    ref = orc.flash_attn_ext(q_u, k, v, pad, scale=scale, q_v=q_v, r=r)
    got = gpu_op(b200, q_u, k, v, pad, scale=scale, q_v=q_v, r=r)
    assert_close(got[:, :valid], ref[:, :valid], "cfg5 fused + padding mask")
    got2 = gpu_op(b200, q_u, k, v, scale=scale, q_v=q_v, r=r, kv_len=[valid])
    assert_close(got2[:, :valid], ref[:, :valid], "cfg5 fused + kv_len")


@pytest.mark.parametrize("T,hd,H", [(200, 128, 8), (611, 128, 8), (150, 64, 4), (97, 80, 4)])
@pytest.mark.parametrize("qdtype", [np.float32, np.float16])
def test_cfg5_position_biases_folded_into_q_load(b200, orc, kernel, T, hd, H, qdtype):
    """Q_u = Q + pos_bias_u and Q_v = Q + pos_bias_v (src/core/fastconformer.h:846-847) formed inside the op
    from one Q: the oracle gets the sums formed ahead of the call in fp32, as the reference's two adds do.
    Q, K and V are views into one fused (T, 3d) projection result, as src/core/fastconformer.h:830-838 builds them."""
    import torch
    rng = np.random.default_rng(46)
    d = H * hd
    qkv = rng.standard_normal((T, 3 * d)).astype(np.float32)
    if qdtype == np.float16:
        qkv = qkv.astype(np.float16).astype(np.float32)
    u = (rng.standard_normal((H, hd)) * 0.3).astype(np.float32)
    vb = (rng.standard_normal((H, hd)) * 0.3).astype(np.float32)
    pe = orc.make_pos_enc(d, T)
    w = (rng.standard_normal((d, d)) / np.sqrt(d)).astype(np.float32)
    r = np.ascontiguousarray((pe @ w).reshape(2 * T - 1, H, hd).transpose(1, 0, 2)[None]).astype(np.float16)

    def heads(x):                                        # (T, d) -> (1, H, T, hd)
        return x.reshape(T, H, hd).transpose(1, 0, 2)[None]

    q, k, v = heads(qkv[:, :d]), heads(qkv[:, d:2 * d]), heads(qkv[:, 2 * d:])
    scale = hd ** -0.5
    ref = orc.flash_attn_ext(q + u[None, :, None], k, v, scale=scale, q_v=q + vb[None, :, None], r=r)

    dev = torch.from_numpy(qkv).cuda()
    if qdtype == np.float16:
        dev = dev.half()

    def dheads(x):
        return x.reshape(T, H, hd).permute(1, 0, 2)[None]  # strided view, no copy

    dq, dk, dv = dheads(dev[:, :d]), dheads(dev[:, d:2 * d]), dheads(dev[:, 2 * d:])
    got = gpu_op(b200, dq, dk, dv, scale=scale, r=r, pos_bias_u=u, pos_bias_v=vb)
    assert_close(got, ref, f"cfg5 folded biases T={T} hd={hd} {np.dtype(qdtype).name}")
    # identical to the two-tensor form when that form is fed the same rounded sums
    q_u = torch.from_numpy(np.ascontiguousarray(q + u[None, :, None])).cuda()
    q_v = torch.from_numpy(np.ascontiguousarray(q + vb[None, :, None])).cuda()
    two = gpu_op(b200, q_u, dk, dv, scale=scale, q_v=q_v, r=r)
    assert np.array_equal(got, two)
    if T == 200:   # the same call with host buffers (bias rows are staged with the other operands)
        hq, hk, hv = (x.cpu() for x in (dq, dk, dv))
        host = b200.flash_attn_ext_host(hq, hk, hv, scale=scale, r=torch.from_numpy(r), pos_bias_u=torch.from_numpy(u),
                                        pos_bias_v=torch.from_numpy(vb)).numpy()
        assert np.array_equal(host, got)


# ---- golden fixtures and edge cases ----------------------------------------------------------------------------------
@pytest.mark.parametrize("name", ["enc64", "gqa128_causal", "perhead_mask", "decode1", "beams5"])
def test_golden_sdpa_fixtures(b200, kernel, name):
    g = np.load(os.path.join(G, "sdpa.npz"))
    mask = g[name + "_mask"] if name + "_mask" in g else None
    got = gpu_op(b200, g[name + "_q"], g[name + "_k"], g[name + "_v"], mask, scale=float(g[name + "_scale"]))
    assert_close(got, g[name + "_out"], name)


def test_golden_cross_attn_kat(b200, kernel):
    """tests/test-core-cross-attn.cpp numbers through the GPU op (hd 4, F32 K/V, unscaled)."""
    g = np.load(os.path.join(G, "crossattn.npz"))
    Q = (g["q_proj"] @ g["dec"]).astype(np.float32).reshape(1, 2, 1, 4)
    got = gpu_op(b200, Q, g["cK"][None], g["cV"][None], scale=1.0)
    # Q, K, V are rounded to F16 on the way to the tensor cores: 1e-3 instead of the test's 1e-4
    assert np.abs(got.reshape(-1) - g["head_out"]).max() < 1e-3


@pytest.mark.parametrize("Tq,Lk,hd,H,Hkv", [(1, 1, 64, 4, 4), (3, 65, 64, 2, 1), (17, 63, 128, 4, 2), (64, 64, 32, 2, 2),
                                           (129, 257, 64, 3, 3), (5, 1000, 128, 8, 8), (100, 7, 128, 2, 2)])
def test_ragged_shapes(b200, orc, kernel, Tq, Lk, hd, H, Hkv):
    rng = np.random.default_rng(Tq * 1000 + Lk)
    q, k, v = randn_f16(rng, (2, H, Tq, hd)), randn_f16(rng, (2, Hkv, Lk, hd)), randn_f16(rng, (2, Hkv, Lk, hd))
    ref = orc.flash_attn_ext(q, k, v, scale=hd ** -0.5)
    assert_close(gpu_op(b200, q, k, v, scale=hd ** -0.5), ref, f"Tq={Tq} Lk={Lk} hd={hd}")


def _random_case(orc, seed):
    """One seeded draw over the op's operand forms; every query row keeps key 0 visible."""
    rng = np.random.default_rng(9000 + seed)
    hd = int(rng.choice([32, 64, 80, 128]))
    kv_kind = str(rng.choice(["f16", "f32", "q8_0"])) if hd % 32 == 0 else str(rng.choice(["f16", "f32"]))
    gqa = int(rng.choice([1, 2, 4]))
    Hkv = int(rng.choice([1, 2, 3]))
    H = Hkv * gqa
    B = int(rng.choice([1, 2, 3]))
    Tq = int(rng.choice([1, 1, 2, 5, 17, 64, 130, 257]))
    Lk = int(rng.integers(Tq, 700)) if rng.random() < 0.5 else int(rng.choice([Tq, 64, 128, 129, 512]))
    Lk = max(Lk, Tq)
    Bk = B if rng.random() < 0.8 else 1
    q = rng.standard_normal((B, H, Tq, hd)).astype(np.float32)
    if rng.random() < 0.5:
        q = q.astype(np.float16)
    x_k = rng.standard_normal((Bk, Hkv, Lk, hd)).astype(np.float32)
    x_v = rng.standard_normal((Bk, Hkv, Lk, hd)).astype(np.float32)
    kw = dict(scale=float(hd ** -0.5 * rng.choice([1.0, 0.5, 2.0])))
    if kv_kind == "q8_0":
        k, v = orc.quantize_q8_0(x_k), orc.quantize_q8_0(x_v)
        kw["kv_type"] = abi.Q8_0
    elif kv_kind == "f16":
        k, v = x_k.astype(np.float16), x_v.astype(np.float16)
    else:
        k, v = x_k, x_v
    mask = None
    form = str(rng.choice(["none", "mask", "causal", "kv_len", "mask+kv_len"]))
    if "mask" in form:
        Hm, Bm = int(rng.choice([1, H])), int(rng.choice([1, B]))
        m = np.where(rng.random((Bm, Hm, Tq, Lk)) < 0.35, -np.inf, 0.0)
        if rng.random() < 0.5:   # finite additive biases as well as -inf
            m = m + np.where(np.isfinite(m), rng.standard_normal(m.shape) * 0.5, 0.0)
        m[..., 0] = 0.0
        mask = m.astype(np.float16)
    if form == "causal":
        kw.update(causal=True, n_past=Lk - Tq)
    if "kv_len" in form:
        kw["kv_len"] = [int(rng.integers(1, Lk + 1)) for _ in range(B)]
    if rng.random() < 0.25:
        kw["softcap"] = float(rng.choice([5.0, 30.0]))
    if mask is not None and rng.random() < 0.3:
        kw["max_bias"] = 8.0
    desc = f"seed {seed}: hd {hd} {kv_kind} q {q.dtype.name} B {B}/{Bk} H {H}/{Hkv} Tq {Tq} Lk {Lk} {form} {sorted(kw)}"
    return q, k, v, mask, kw, desc


@pytest.mark.parametrize("seed", range(96))
def test_random_operand_forms(b200, orc, seed):
    """Seeded sweep over head dims, GQA ratios, batch broadcast, K/V types, mask shapes, causal bound, device
    kv_len, softcap and ALiBi, with the automatic kernel choice and with the general tile kernel forced."""
    import torch
    q, k, v, mask, kw, desc = _random_case(orc, seed)
    ref = orc.flash_attn_ext(q.astype(np.float32), k, v, mask, **kw)
    dk, dv = k, v
    if seed % 2:   # token-major cache rows (Bk, Lk, Hkv, row) read through a head-major strided view
        dk = torch.from_numpy(np.ascontiguousarray(k.transpose(0, 2, 1, 3))).cuda().permute(0, 2, 1, 3)
        dv = torch.from_numpy(np.ascontiguousarray(v.transpose(0, 2, 1, 3))).cuda().permute(0, 2, 1, 3)
        desc += " token-major K/V"
    for kern in (abi.KERNEL_NONE, abi.KERNEL_TILE_MMA):
        assert b200.lib().b200_set_kernel_override(kern) == 0
        try:
            got = gpu_op(b200, q, dk, dv, mask, **kw)
        finally:
            b200.lib().b200_set_kernel_override(abi.KERNEL_NONE)
        assert_close(got, ref, f"{desc} override {kern}")


def test_f32_kv_softcap_alibi(b200, orc, kernel):
    rng = np.random.default_rng(8)
    q = randn_f16(rng, (1, 6, 70, 64)).astype(np.float32)
    k = randn_f16(rng, (1, 6, 90, 64)).astype(np.float32)
    v = randn_f16(rng, (1, 6, 90, 64)).astype(np.float32)
    m = (rng.standard_normal((1, 1, 70, 90))).astype(np.float16)
    ref = orc.flash_attn_ext(q, k, v, m, scale=0.3, max_bias=8.0, softcap=5.0)
    assert_close(gpu_op(b200, q, k, v, m, scale=0.3, max_bias=8.0, softcap=5.0), ref, "F32 KV + softcap + ALiBi")


def test_fully_masked_rows_and_empty_cache(b200, orc, kernel):
    rng = np.random.default_rng(6)
    q, k, v = randn_f16(rng, (2, 4, 9, 64)), randn_f16(rng, (2, 4, 80, 64)), randn_f16(rng, (2, 4, 80, 64))
    m = np.zeros((1, 1, 9, 80), np.float16)
    m[0, 0, 4, :] = -np.inf
    ref = orc.flash_attn_ext(q, k, v, m, scale=0.125)
    got = gpu_op(b200, q, k, v, m, scale=0.125)
    assert np.all(got[:, 4] == 0)
    assert_close(got, ref, "fully masked row")
    got = gpu_op(b200, q, k, v, scale=0.125, kv_len=[0, 80])
    assert np.all(got[0] == 0)
    assert_close(got, orc.flash_attn_ext(q, k, v, scale=0.125, kv_len=[0, 80]), "kv_len 0")


def test_host_buffer_entry_point(b200, orc):
    rng = np.random.default_rng(12)
    q = torch.from_numpy(randn_f16(rng, (2, 8, 5, 64)).astype(np.float32)).pin_memory()
    k = torch.from_numpy(randn_f16(rng, (2, 8, 300, 64))).pin_memory()
    v = torch.from_numpy(randn_f16(rng, (2, 8, 300, 64))).pin_memory()
    out = b200.flash_attn_ext_host(q, k, v, scale=0.125, kv_len=torch.tensor([300, 123], dtype=torch.int32))
    ref = orc.flash_attn_ext(q.numpy(), k.numpy(), v.numpy(), scale=0.125, kv_len=[300, 123])
    assert_close(out.numpy(), ref, "host entry point")
    b200.lib().b200_host_arena_release()


def test_host_entry_point_chunked_decode_workspace(b200, orc):
    """A decode batch large enough for one KV split per (stream, head) as a whole, but split when the host entry
    point pipelines it in four batch chunks: the chunk launches need more split workspace than the whole call
    would.  The chunked host result must equal the one-launch device result."""
    rng = np.random.default_rng(77)
    B, H, Lk, hd = 80, 8, 300, 64
    q = torch.from_numpy(randn_f16(rng, (B, H, 1, hd))).pin_memory()
    k = torch.from_numpy(randn_f16(rng, (B, H, Lk, hd))).pin_memory()
    v = torch.from_numpy(randn_f16(rng, (B, H, Lk, hd))).pin_memory()
    out = b200.flash_attn_ext_host(q, k, v, scale=0.125)
    dev = b200.flash_attn_ext(q.cuda(), k.cuda(), v.cuda(), scale=0.125)
    torch.cuda.synchronize()
    assert b200.lib().b200_last_kernel() == abi.KERNEL_DECODE_SPLIT
    assert float((out - dev.cpu()).abs().max()) < 1e-3   # same kernel; split count differs (summation order, f16 rounding of P against another reference maximum)
    for b in (0, 79):
        ref = orc.flash_attn_ext(q[b:b + 1].numpy(), k[b:b + 1].numpy(), v[b:b + 1].numpy(), scale=0.125)
        assert_close(out[b:b + 1].numpy(), ref, f"chunked host decode, stream {b}")
    b200.lib().b200_host_arena_release()


def test_full_size_properties_cfg3(b200, orc):
    """Full size of the Whisper large-v3 encoder workload (64 segments x 20 heads x 1500 frames, one layer): two sampled
    segments against the oracle, batch invariance (a segment computed inside the batch equals the same segment
    computed alone, bit for bit), softmax weights summing to one (V = ones), and linearity in V."""
    gen = torch.Generator(device="cuda").manual_seed(2)
    S, H, T, hd = 64, 20, 1500, 64
    q, k, v = (torch.randn((S, H, T, hd), generator=gen, device="cuda", dtype=torch.float32).half() for _ in range(3))
    out = b200.flash_attn_ext(q, k, v, scale=0.125)
    torch.cuda.synchronize()
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5 and b200.lib().b200_device_status() == 0
    for seg in (0, 41):
        ref = orc.flash_attn_ext(q[seg:seg + 1].cpu().numpy(), k[seg:seg + 1].cpu().numpy(), v[seg:seg + 1].cpu().numpy(), scale=0.125)
        assert_close(out[seg:seg + 1].cpu().numpy(), ref, f"cfg3 full batch, segment {seg}")
        alone = b200.flash_attn_ext(q[seg:seg + 1], k[seg:seg + 1], v[seg:seg + 1], scale=0.125)
        assert torch.equal(alone[0], out[seg]), "a segment's result must not depend on its batch neighbours"
    ones = b200.flash_attn_ext(q, k, torch.ones_like(v), scale=0.125)
    assert float((ones - 1.0).abs().max()) < 2e-3
    v2 = torch.randn((S, H, T, hd), generator=gen, device="cuda", dtype=torch.float32).half()
    lin = b200.flash_attn_ext(q[:4], k[:4], (v[:4].float() * 0.5 + v2[:4].float() * 0.25).half(), scale=0.125)
    want = 0.5 * out[:4] + 0.25 * b200.flash_attn_ext(q[:4], k[:4], v2[:4], scale=0.125)
    assert float((lin - want).abs().max()) < 4e-3   # V is re-rounded to f16 after the combination


def test_full_size_properties_cfg5(b200, orc, capsys):
    """Full size of the FastConformer workload (T = 7500, 8 heads, hd 128) at the path's own tolerance: 97 query rows
    that cover more than 64 different positions inside a 128-row tile (and both ends of the sequence) against the
    oracle's rel-pos path restricted to those rows, with the measured errors printed and attributed against the
    fp64 run; plus the size-independent property that softmax weights sum to one (V = ones gives ones)."""
    rng = np.random.default_rng(4)
    T = 7500
    q_u, q_v, k, v, r = _relpos_case(orc, rng, T)
    scale = 128 ** -0.5
    got = gpu_op(b200, q_u, k, v, scale=scale, q_v=q_v, r=r)
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5 and b200.lib().b200_device_status() == 0
    rows = sorted({128 * ((i * 11) % 58) + (4 * i) // 3 for i in range(96)} | {0, 1, 63, 64, 127, 128, 3749, 7437, 7499})
    assert len(rows) >= 64 and len({x % 128 for x in rows}) >= 64
    ref = orc.flash_attn_ext(q_u, k, v, scale=scale, q_v=q_v, r=r, rows=rows)
    gold = orc.flash_attn_ext(q_u, k, v, scale=scale, q_v=q_v, r=r, rows=rows, gold=True)
    e_gpu, e_gold, e_orc = errors(got[:, rows], ref[:, rows]), errors(got[:, rows], gold[:, rows]), errors(ref[:, rows], gold[:, rows])
    with capsys.disabled():
        print(f"\n  cfg5 T={T}, {len(rows)} rows: GPU vs oracle max-abs {e_gpu[0]:.3e} rel-L2 {e_gpu[1]:.3e}; "
              f"GPU vs fp64 {e_gold[0]:.3e} / {e_gold[1]:.3e}; oracle fp32 vs fp64 {e_orc[0]:.3e} / {e_orc[1]:.3e}")
    assert_close(got[:, rows], ref[:, rows], "cfg5 full size, sampled rows")
    ones = np.ones_like(v)
    got1 = gpu_op(b200, q_u, k, ones, scale=scale, q_v=q_v, r=r)
    assert np.abs(got1 - 1.0).max() < 2e-3


@pytest.mark.parametrize("T", [200, 611])
def test_cfg5_relpos_with_explicit_masks_on_the_tensor_core_path(b200, orc, T):
    """The fused bias combined with an explicit F16 mask stays on the tcgen05 kernel: the bucket padding mask of
    src/canary_ctc.cpp:370-382 (pad keys -inf), the local-attention window of src/core/fastconformer.h:887-895
    (a band of width 2*64+1, -inf outside), and a per-head finite mask; a query row whose window is empty of valid
    keys gives zeros."""
    rng = np.random.default_rng(45)
    q_u, q_v, k, v, r = _relpos_case(orc, rng, T)
    scale = 128 ** -0.5
    valid = T - 29
    pad = np.zeros((1, 1, T, T), np.float16)
    pad[..., valid:] = -np.inf
    qi, ki = np.arange(T)[:, None], np.arange(T)[None, :]
    band = np.where(np.abs(qi - ki) <= 64, 0.0, -np.inf).astype(np.float16)[None, None]
    per_head = (rng.standard_normal((1, 8, T, T)) * 0.5).astype(np.float16)
    per_head[0, 3, 17, :] = -np.inf                      # one fully masked row
    for name, mask in (("padding", pad), ("local window", band), ("padding + window", (pad.astype(np.float32) + band).astype(np.float16)),
                       ("per-head", per_head)):
        ref = orc.flash_attn_ext(q_u, k, v, mask, scale=scale, q_v=q_v, r=r)
        got = gpu_op(b200, q_u, k, v, mask, scale=scale, q_v=q_v, r=r)
        assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5, name
        rows = slice(0, valid) if "padding" in name else slice(0, T)
        assert_close(got[:, rows], ref[:, rows], f"cfg5 fused bias + {name} mask, T={T}")
    assert not gpu_op(b200, q_u, k, v, per_head, scale=scale, q_v=q_v, r=r)[0, 17, 3].any()
    assert b200.lib().b200_device_status() == 0


@pytest.mark.parametrize("T", [1, 2, 63, 64, 65, 127, 128, 129, 191, 193, 256, 257, 385, 640])
@pytest.mark.parametrize("spread", [1.0, 4.0])
def test_relpos_edges_of_tiles_and_growing_scores(b200, orc, T, spread):
    """Sizes around the kernel's 64-column blocks and 128-key tiles; keys scaled by 4 make scores outgrow the reference of the
    running softmax in later tiles."""
    rng = np.random.default_rng(461)
    q_u, q_v, k, v, r = _relpos_case(orc, rng, T, H=2, d_model=256)
    k *= np.float32(spread)
    ref = orc.flash_attn_ext(q_u, k, v, scale=128 ** -0.5, q_v=q_v, r=r)
    got = gpu_op(b200, q_u, k, v, scale=128 ** -0.5, q_v=q_v, r=r)
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5
    assert_close(got, ref, f"rel-pos T={T} spread={spread}")
    assert b200.lib().b200_device_status() == 0


@pytest.mark.parametrize("T", [136, 140, 142, 141, 264, 267])
def test_relpos_mask_rows_of_every_alignment(b200, orc, T):
    """Mask rows on 16-, 8-, 4- and 2-byte boundaries, with a partial last tile."""
    rng = np.random.default_rng(462)
    q_u, q_v, k, v, r = _relpos_case(orc, rng, T, H=2, d_model=256)
    qi, ki = np.arange(T)[:, None], np.arange(T)[None, :]
    mask = (np.where(np.abs(qi - ki) <= 40, 0.0, -np.inf) + rng.standard_normal((T, T)) * 0.5).astype(np.float16)[None, None]
    ref = orc.flash_attn_ext(q_u, k, v, mask, scale=128 ** -0.5, q_v=q_v, r=r)
    got = gpu_op(b200, q_u, k, v, mask, scale=128 ** -0.5, q_v=q_v, r=r)
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5
    assert_close(got, ref, f"rel-pos with a mask, T={T}")
    assert b200.lib().b200_device_status() == 0


@pytest.mark.parametrize("scale", [2.0 ** -16, 0.04, 0.125, 1.0, 2.0 ** 14])
def test_relpos_scales(b200, orc, scale):
    """Scales that are powers of two, are not, or lie outside the range of the tensor-core kernel (the general kernel takes those)."""
    rng = np.random.default_rng(463)
    q_u, q_v, k, v, r = _relpos_case(orc, rng, 150, H=2, d_model=256)
    f = np.float32(min(1.0, 128 ** -0.5 / scale))   # scores of ordinary size also under a large scale
    q_u, q_v = (q_u * f).astype(np.float16).astype(np.float32), (q_v * f).astype(np.float16).astype(np.float32)
    ref = orc.flash_attn_ext(q_u, k, v, scale=scale, q_v=q_v, r=r)
    got = gpu_op(b200, q_u, k, v, scale=scale, q_v=q_v, r=r)
    assert (b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5) == (2.0 ** -14 <= scale <= 2.0 ** 13)
    assert_close(got, ref, f"rel-pos scale={scale}")


@pytest.mark.parametrize("size", [4.0, 8.0, 16.0])
@pytest.mark.parametrize("T", [150, 700])
def test_relpos_bias_of_any_size_is_rounded_once(b200, orc, T, size):
    """f16(scale * x) of a bias of standard deviation `size`: a step of F16 grows with it, so that a rounding elsewhere than the
    operator's (of x / d, say, times d afterwards) shows."""
    rng = np.random.default_rng(464)
    q_u, q_v, k, v, r = _relpos_case(orc, rng, T, H=2, d_model=256)
    r = (r.astype(np.float32) * np.float32(size / orc.relpos_mask(q_v, r, 128 ** -0.5).astype(np.float32).std())).astype(np.float16)
    ref = orc.flash_attn_ext(q_u, k, v, scale=128 ** -0.5, q_v=q_v, r=r)
    got = gpu_op(b200, q_u, k, v, scale=128 ** -0.5, q_v=q_v, r=r)
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5
    assert_close(got, ref, f"rel-pos T={T} bias of {size}")
    assert b200.lib().b200_device_status() == 0


@pytest.mark.parametrize("T,valid", [(150, 131), (300, 257), (300, 127), (100, 3)])
def test_relpos_table_rows_of_dead_keys_hold_anything(b200, orc, T, valid):
    """Rows of the table that only keys at or beyond kv_len reach (bucket padding) hold NaN: no living key sees them."""
    rng = np.random.default_rng(465)
    q_u, q_v, k, v, r = _relpos_case(orc, rng, T, H=2, d_model=256)
    pad = np.zeros((1, 1, T, T), np.float16)
    pad[..., valid:] = -np.inf
    ref = orc.flash_attn_ext(q_u, k, v, pad, scale=128 ** -0.5, q_v=q_v, r=r)
    r[:, :, T - 1 + valid:] = np.nan
    got = gpu_op(b200, q_u, k, v, scale=128 ** -0.5, q_v=q_v, r=r, kv_len=[valid])
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5
    assert_close(got, ref, f"rel-pos T={T} kv_len={valid}")
    assert b200.lib().b200_device_status() == 0


@pytest.mark.parametrize("T", [200, 330])
def test_relpos_batch_of_lengths_around_the_blocks(b200, orc, T):
    """Utterances whose last tiles hold 64 query rows or keys or fewer, which leave out blocks of 64 table rows, and of one row or key more;
    their lengths for queries and keys need not be the same."""
    rng = np.random.default_rng(467)
    lens = [n for n in (1, 63, 64, 65, 128, 129, 191, 192, 193, 200, 256, 257, 320, 321, 330) if n <= T]
    qlens, klens = lens + lens, lens + lens[::-1]
    q_u, q_v, k, v, r = _relpos_case(orc, rng, T, H=2, d_model=256)
    B = len(qlens)
    roll = lambda x: np.concatenate([np.roll(x, 7 * b, axis=2) for b in range(B)])
    q_u, q_v, k, v = (roll(x) for x in (q_u, q_v, k, v))
    got = gpu_op(b200, q_u, k, v, scale=128 ** -0.5, q_v=q_v, r=r, q_len=qlens, kv_len=klens)
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5 and b200.lib().b200_device_status() == 0
    for b, (nq, nk) in enumerate(zip(qlens, klens)):
        pad = np.zeros((1, 1, T, T), np.float16)
        pad[..., nk:] = -np.inf
        one = slice(b, b + 1)
        ref = orc.flash_attn_ext(q_u[one], k[one], v[one], pad, scale=128 ** -0.5, q_v=q_v[one], r=r)
        assert_close(got[one, :nq], ref[:, :nq], f"rel-pos T={T} q_len={nq} kv_len={nk}")
        assert not got[b, nq:].any()


def test_relpos_bias_beyond_f16_is_an_infinity(b200, orc):
    """A bias of -inf (scale * x below the range of F16) removes its key, and that key only; one just inside the range is itself."""
    rng = np.random.default_rng(466)
    T = 200
    q_u, q_v, k, v, r = _relpos_case(orc, rng, T, H=2, d_model=256)
    q_v[..., 0] = 16.0
    for distance, x in ((5, -60000.0), (-31, -60000.0), (70, -46000.0)):   # scale * 16 * x: -84853 (twice) and -65054
        r[:, :, T - 1 + distance] = 0.0
        r[:, :, T - 1 + distance, 0] = x
    bias = orc.relpos_mask(q_v, r, 128 ** -0.5)
    assert np.isneginf(bias).sum() == 2 * (T - 5 + T - 31) and not np.isnan(bias).any()
    ref = orc.flash_attn_ext(q_u, k, v, scale=128 ** -0.5, q_v=q_v, r=r)
    got = gpu_op(b200, q_u, k, v, scale=128 ** -0.5, q_v=q_v, r=r)
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5
    assert_close(got, ref, "rel-pos with biases of -inf")
    # query 10: every key removed but one
    r[:] = 0.0
    r[:, :, :, 0] = -60000.0
    r[:, :, T - 1 + 7, 0] = 0.0
    got = gpu_op(b200, q_u, k, v, scale=128 ** -0.5, q_v=q_v, r=r)
    assert_close(got[0, 10], v[0, :, 17], "one key left", max_abs=0.0, rel_l2=0.0)
    assert not got[0, T - 1].any()                       # no key left: zeros, as under a mask
    assert b200.lib().b200_device_status() == 0


def test_relpos_table_built_on_the_device_and_cached(b200, orc):
    """R = attn_pos_w . pos_enc (src/core/fastconformer.h:118-130, :843, :851) built by the library for a (layer, T)
    equals the oracle's make_pos_enc @ W to within one F16 rounding, attention with the library's table meets the
    parity tolerance against the oracle with the host-built table, and the cache returns the same table for the
    same key, builds per T, and evicts the least recently used entry."""
    import ctypes as C
    rng = np.random.default_rng(47)
    T, H, hd = 333, 8, 128
    d = H * hd
    w = (rng.standard_normal((d, d)) / 32.0).astype(np.float32)          # numpy (d_out, d_in) == ggml [d_in, d_out]
    r_host = (orc.make_pos_enc(d, T) @ w.T).reshape(2 * T - 1, H, hd).transpose(1, 0, 2)   # (H, 2T-1, hd)
    L = b200.lib()
    cache = C.c_void_p()
    assert L.b200_relpos_cache_create(2, 2, C.byref(cache)) == 0
    st = torch.cuda.current_stream().cuda_stream
    for wt, tol in ((torch.from_numpy(w).cuda(), 1.0), (torch.from_numpy(w).cuda().half(), 1.0)):
        tw, tr, hit = abi.from_torch(wt), abi.Tensor(), C.c_int(-1)
        assert L.b200_relpos_cache_get(cache, 0, T, C.byref(tw), H, st, C.byref(tr), C.byref(hit)) == 0 and hit.value == 0
        assert (tr.ne[0], tr.ne[1], tr.ne[2], tr.type) == (hd, 2 * T - 1, H, abi.F16) and tr.data % 16 == 0
        torch.cuda.synchronize()
        got = torch.empty((H, 2 * T - 1, hd), dtype=torch.float16, device="cuda")
        C.cdll.LoadLibrary("libcudart.so").cudaMemcpy(C.c_void_p(got.data_ptr()), C.c_void_p(tr.data), C.c_size_t(got.numel() * 2), 3)
        want = (orc.make_pos_enc(d, T) @ wt.float().cpu().numpy().T).reshape(2 * T - 1, H, hd).transpose(1, 0, 2)
        diff = np.abs(got.float().cpu().numpy() - want)
        ulp = 2.0 ** (np.floor(np.log2(np.maximum(np.abs(want), 2.0 ** -14))) - 10)      # one F16 ulp at each value
        # one F16 rounding, plus the fp32 summation-order noise of a 1024-term dot product (and, for the F16 weight,
        # nothing more: the weight is widened exactly)
        assert (diff <= tol * ulp + 4e-6).all(), f"table differs by {float(((diff - 4e-6) / ulp).max()):.2f} F16 ulp"
        tr2 = abi.Tensor()
        assert L.b200_relpos_cache_get(cache, 0, T, C.byref(tw), H, st, C.byref(tr2), C.byref(hit)) == 0 and hit.value == 1
        assert tr2.data == tr.data
    # attention with the library-built table (F32 weight entry was evicted? no: two entries per layer, both alive)
    q_u = rng.standard_normal((1, H, T, hd)).astype(np.float16).astype(np.float32)
    q_v = rng.standard_normal((1, H, T, hd)).astype(np.float16).astype(np.float32)
    k, v = randn_f16(rng, (1, H, T, hd)), randn_f16(rng, (1, H, T, hd))
    ref = orc.flash_attn_ext(q_u, k, v, scale=hd ** -0.5, q_v=q_v, r=np.ascontiguousarray(r_host[None]).astype(np.float16))
    wt = torch.from_numpy(w).cuda()
    tw, tr, hit = abi.from_torch(wt), abi.Tensor(), C.c_int(-1)
    assert L.b200_relpos_cache_get(cache, 1, T, C.byref(tw), H, st, C.byref(tr), C.byref(hit)) == 0 and hit.value == 0
    r_dev = torch.empty((1, H, 2 * T - 1, hd), dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    C.cdll.LoadLibrary("libcudart.so").cudaMemcpy(C.c_void_p(r_dev.data_ptr()), C.c_void_p(tr.data), C.c_size_t(r_dev.numel() * 2), 3)
    got = gpu_op(b200, q_u, k, v, scale=hd ** -0.5, q_v=q_v, r=r_dev)
    assert_close(got, ref, "attention with the device-built table")
    # eviction: a third and fourth T on layer 1 push out the oldest entries; bytes follow
    for T2 in (40, 50, 60):
        assert L.b200_relpos_cache_get(cache, 1, T2, C.byref(tw), H, st, C.byref(tr), C.byref(hit)) == 0 and hit.value == 0
    assert L.b200_relpos_cache_get(cache, 1, T, C.byref(tw), H, st, C.byref(tr), C.byref(hit)) == 0 and hit.value == 0   # was evicted
    assert L.b200_relpos_cache_get(cache, 1, 60, C.byref(tw), H, st, C.byref(tr), C.byref(hit)) == 0 and hit.value == 1
    assert L.b200_relpos_cache_bytes(cache) == 2 * d * (2 * T - 1) * 2 + d * (2 * T - 1) * 2 + d * (2 * 60 - 1) * 2
    assert L.b200_relpos_cache_get(cache, 5, T, C.byref(tw), H, st, C.byref(tr), None) == abi.E_SHAPE
    torch.cuda.synchronize()
    L.b200_relpos_cache_destroy(cache)


def test_launch_tracing_records_one_event_pair_per_launch(b200, orc):
    """b200_trace_enable / b200_trace_read: every launch is bracketed by an event pair (and an NVTX range); records
    come back oldest first with the launch's geometry and a positive device time; a full ring keeps the newest."""
    import ctypes as C
    L = b200.lib()
    rng = np.random.default_rng(60)
    assert L.b200_trace_enable(4) == 0
    try:
        qp, kp = randn_f16(rng, (1, 4, 300, 64)), randn_f16(rng, (1, 4, 300, 64))
        qd, kd = randn_f16(rng, (2, 8, 1, 128)), randn_f16(rng, (2, 2, 700, 128))
        got = gpu_op(b200, qp, kp, kp, scale=0.125)
        gpu_op(b200, qd, kd, kd, scale=0.1)
        recs, n = (abi.TraceRecord * 8)(), C.c_int(0)
        assert L.b200_trace_read(recs, 8, C.byref(n)) == 0 and n.value == 2
        assert (recs[0].kernel, recs[0].head_dim, recs[0].q_len, recs[0].kv_len, recs[0].n_heads, recs[0].n_batch) == (abi.KERNEL_PREFILL_TC5, 64, 300, 300, 4, 1)
        assert (recs[1].kernel, recs[1].head_dim, recs[1].q_len, recs[1].kv_len, recs[1].n_kv_heads, recs[1].n_batch) == (abi.KERNEL_DECODE_SPLIT, 128, 1, 700, 2, 2)
        assert recs[1].n_splits >= 1 and 0.0 < recs[0].ms < 50.0 and 0.0 < recs[1].ms < 50.0
        assert L.b200_trace_read(recs, 8, C.byref(n)) == 0 and n.value == 0       # read clears
        for _ in range(6):                                                        # ring of 4: the two oldest are dropped
            gpu_op(b200, qd, kd, kd, scale=0.1)
        assert L.b200_trace_read(recs, 8, C.byref(n)) == 0 and n.value == 4
        assert_close(got, orc.flash_attn_ext(qp, kp, kp, scale=0.125), "traced launch")   # tracing does not change results
    finally:
        assert L.b200_trace_enable(0) == 0
    gpu_op(b200, qd, kd, kd, scale=0.1)
    n = C.c_int(5)
    assert L.b200_trace_read(None, 0, C.byref(n)) == 0 and n.value == 0


@pytest.mark.parametrize("hd,Hkv,gqa", [(128, 8, 4), (128, 7, 1), (128, 8, 8)])
@pytest.mark.parametrize("L", [130, 257, 400])
def test_q8_0_decode_wide_ctas(b200, orc, hd, Hkv, gqa, L):
    """Between the unit counts that clusters fill and those that fill the SMs one CTA of eight warps takes a (stream, KV
    head) whole, in tiles of 128 keys: lengths around the edges of a tile and of a warp's 16 keys, an empty stream, one to
    eight query rows per KV head."""
    rng = np.random.default_rng(hd + L + gqa)
    B = 34
    q = randn_f16(rng, (B, Hkv * gqa, 1, hd))
    k, v = (orc.quantize_q8_0(rng.standard_normal((B, Hkv, L, hd)).astype(np.float32)) for _ in "kv")
    lens = rng.integers(1, L + 1, B).astype(np.int32)
    edges = [0, 1, 15, 16, 17, 127, 128, 129, L]
    lens[:len(edges)] = np.minimum(edges, L)
    kw = dict(scale=hd ** -0.5, kv_type=abi.Q8_0, kv_len=lens)
    ctx = -(-L // 32) * 32                       # rows per head as the slabs lay them out: 16-byte aligned heads
    slabs = [np.zeros((B, Hkv, ctx, x.shape[-1]), np.uint8) for x in (k, v)]
    for s, x in zip(slabs, (k, v)):
        s[:, :, :L] = x
    dk, dv = (cuda_view(s[:, :, :L], s) for s in slabs)
    assert b200.plan(torch.from_numpy(q), dk, dv, scale=1.0, kv_type=abi.Q8_0) == (abi.KERNEL_DECODE_SPLIT, 1)
    assert_close(gpu_op(b200, q, dk, dv, **kw), orc.flash_attn_ext(q, k, v, **kw), f"wide decode hd={hd} L={L}")
    assert b200.lib().b200_device_status() == 0


@pytest.mark.parametrize("T,H,gqa", [(700, 6, 1), (1000, 4, 2), (1473, 3, 1), (2050, 1, 1)])
@pytest.mark.parametrize("form", ["plain", "causal", "lengths"])
@pytest.mark.parametrize("q_f32", [False, True])
def test_prefill_shared_query_tiles(b200, orc, T, H, gqa, form, q_f32):
    """Few query tiles of head_dim 64 over many keys: the key steps of a tile are shared by the CTAs of a cluster (two to
    eight).  Step counts that do not divide, tiles of which some CTAs see no key (causal, ragged lengths, an empty entry),
    grouped heads, rows whose maximum moves far while the steps go by."""
    rng = np.random.default_rng(T + H + q_f32)
    B, Hkv = (2, H // gqa) if form == "lengths" else (1, H // gqa)
    q, k, v = randn_f16(rng, (B, H, T, 64)), randn_f16(rng, (B, Hkv, T, 64)), randn_f16(rng, (B, Hkv, T, 64))
    q[:, 0] *= 6.0
    if q_f32:
        q = q.astype(np.float32)
    kw = dict(scale=0.125)
    if form == "causal":
        kw.update(causal=True, n_past=0)
    if form == "lengths":
        kw.update(kv_len=np.array([T, 70], np.int32), q_len=np.array([T - 1, 40], np.int32))
    got = gpu_op(b200, q, k, v, **kw)
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5
    q_len = kw.pop("q_len", None)
    ref = orc.flash_attn_ext(q, k, v, **kw)
    if q_len is not None:
        for b, n in enumerate(q_len):
            ref[b, n:] = 0.0
    assert_close(got, ref, f"shared tiles T={T} H={H} gqa={gqa} {form}")
    assert b200.lib().b200_device_status() == 0


@pytest.mark.parametrize("B,H,Hkv,Tq,Lk,hd", [(1, 20, 20, 1500, 1500, 64), (2, 16, 4, 1100, 1100, 128), (3, 8, 2, 300, 1300, 128), (2, 20, 20, 5, 1500, 64), (1, 6, 6, 650, 650, 80)])
@pytest.mark.parametrize("q_f32", [False, True])
def test_host_entry_point_pinned_result(b200, orc, B, H, Hkv, Tq, Lk, hd, q_f32):
    """A pinned result is written by the kernels and lets the call run over chunks of heads: one to three entries, grouped
    heads, each kernel family (head dims 64 and 128 on the tensor path, decode rows, a padded head dim), lengths per entry;
    a pageable result of the same operands is staged and must agree."""
    rng = np.random.default_rng(B * 1000 + H + hd)
    q = randn_f16(rng, (B, H, Tq, hd))
    k, v = (randn_f16(rng, (B, Hkv, Lk, hd)) for _ in "kv")
    lens = np.array([Lk, 17, Lk - 1][:B], np.int32)
    kw = dict(scale=hd ** -0.5, kv_len=torch.from_numpy(lens))
    args = [torch.from_numpy(x.astype(np.float32) if q_f32 and i == 0 else x).pin_memory() for i, x in enumerate((q, k, v))]
    out = torch.full((B, Tq, H, hd), float("nan"), dtype=torch.float32).pin_memory()
    assert b200.flash_attn_ext_host(*args, out=out, **kw) is out
    ref = orc.flash_attn_ext(q, k, v, scale=hd ** -0.5, kv_len=lens)
    assert_close(out.numpy(), ref, "host entry point, pinned result")
    assert_close(b200.flash_attn_ext_host(*args, **kw).numpy(), ref, "host entry point, pageable result")


@pytest.mark.parametrize("T,H", [(256, 6), (1000, 4)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("pos", [14, 15, 20, 30, 63, 78, 79, 94, 255])
def test_prefill_one_key_far_above_the_others(b200, orc, T, H, causal, pos):
    """head_dim 64 prefill with one key 60 to 400 nats above all others (the log2-domain distance passes 127, where a float's
    exponent ends), in each kind of column of the first and of a later 64-key step; T = 256 with a CTA per query tile,
    T = 1000 with the key steps shared by a cluster.  Every row that sees the key is that key's value row."""
    gaps = [60.0, 88.9, 95.0, 120.0, 200.0, 400.0]
    for lo in range(0, len(gaps), H):
        part = gaps[lo:lo + H]
        rng = np.random.default_rng(pos + T)
        n = len(part)
        q = (1.0 + 0.01 * rng.standard_normal((1, n, T, 64))).astype(np.float16)
        k, v = randn_f16(rng, (1, n, T, 64), 0.01), randn_f16(rng, (1, n, T, 64))
        k[0, :, pos] = (np.array(part) / (0.125 * 64))[:, None].astype(np.float16)   # score = gap (1 +- 0.01)
        kw = dict(scale=0.125, causal=causal)
        got = gpu_op(b200, q, k, v, **kw)
        assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5
        assert_close(got, orc.flash_attn_ext(q, k, v, **kw), f"key {pos} {part} nats above, T={T} causal={causal}")
        # all other keys together weigh less than T e^-59 of it: the row is V[pos], |V| < 5, times P / l.  The key's score in
        # the log2 domain (at most 590) is exact in the product but rounded as the reference (2^-15): l is 1 to 2.2e-5
        seen = slice(pos, T) if causal else slice(0, T)
        assert np.abs(got[0, seen] - v[0, :, pos].astype(np.float32)[None]).max() <= 5 * 2.2e-5 + 1e-5
    assert b200.lib().b200_device_status() == 0


@pytest.mark.parametrize("T,H", [(256, 6), (1000, 4)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("pos", [14, 20, 31, 79, 255])
def test_prefill_keeps_a_nan(b200, T, H, causal, bad, pos):
    """A key row of NaN, or of +inf against positive query rows (inf - inf), in each kind of column of a key step: every row
    that sees the key is NaN, every other row is finite."""
    rng = np.random.default_rng(pos + T)
    q = np.abs(randn_f16(rng, (1, H, T, 64))) + np.float16(0.1)
    k, v = randn_f16(rng, (1, H, T, 64)), randn_f16(rng, (1, H, T, 64))
    k[0, :, pos] = bad
    got = gpu_op(b200, q, k, v, scale=0.125, causal=causal)
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5
    first = pos if causal else 0
    assert np.isnan(got[0, first:]).all()
    assert np.isfinite(got[0, :first]).all()
    assert b200.lib().b200_device_status() == 0


@pytest.mark.parametrize("hidden", [16, 64, 128, 200])
@pytest.mark.parametrize("T", [300, 1000])
def test_prefill_low_scores_behind_keys_of_minus_infinity(b200, orc, hidden, T):
    """The first keys of every row score -inf, the others about -100: they carry the row although none of them would be seen
    against a reference of 0 (2^-144)."""
    rng = np.random.default_rng(hidden + T)
    q = (1.0 + 0.02 * rng.standard_normal((1, 4, T, 64))).astype(np.float16)
    k, v = (-12.5 + 0.02 * rng.standard_normal((1, 4, T, 64))).astype(np.float16), randn_f16(rng, (1, 4, T, 64))
    k[:, :, :hidden] = -np.inf
    got = gpu_op(b200, q, k, v, scale=0.125)
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5
    assert_close(got, orc.flash_attn_ext(q, k, v, scale=0.125), f"{hidden} keys of -inf, T={T}")
    assert b200.lib().b200_device_status() == 0


@pytest.mark.parametrize("hidden", [64, 128, 200])
@pytest.mark.parametrize("low", ["scores", "mask"])
def test_relpos_low_scores_behind_masked_keys(b200, orc, hidden, low):
    """Fused bias with an explicit mask whose first keys are -inf, the others' scores about -100, or their mask the lowest
    finite F16: the visible keys carry the row."""
    rng = np.random.default_rng(hidden)
    T = 400
    q_u, q_v, k, v, r = _relpos_case(orc, rng, T)
    mask = np.zeros((1, 1, T, T), np.float16)
    if low == "scores":
        # (F16 numbers in whatever type: the kernels round F32 keys to F16, at this size by more than the tolerance)
        q_u = (1.0 + 0.02 * rng.standard_normal(q_u.shape)).astype(np.float16).astype(q_u.dtype)
        k = (-100.0 / 128 ** 0.5 + 0.02 * rng.standard_normal(k.shape)).astype(np.float16).astype(k.dtype)
    else:
        mask[:] = np.finfo(np.float16).min
    mask[..., :hidden] = -np.inf
    kw = dict(scale=128 ** -0.5, q_v=q_v, r=r)
    got = gpu_op(b200, q_u, k, v, mask, **kw)
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5
    ref = orc.flash_attn_ext(q_u, k, v, mask, **kw)
    # against a mask of -65504 a logit is rounded to 2^-8 (the sum in fp32): 0.4 % of P
    assert_close(got, ref, f"{low} behind {hidden} masked keys", **(dict(max_abs=2e-2, rel_l2=1e-2) if low == "mask" else {}))
    assert b200.lib().b200_device_status() == 0


@pytest.mark.parametrize("form", ["hd64", "hd64 shared", "relpos"])
@pytest.mark.parametrize("pos", [30, 80, 200])
def test_prefill_rounds_no_weight_of_a_row_that_one_key_carries(b200, form, pos):
    """Key 0 stands 2^8.2 to 2^11.9 below key `pos` and everything else e^-30 below key 0: key `pos` carries the row and its P
    has to be exact.  What may be wrong is the F16 rounding of key 0's P (2^-12 of 2^-8.2) and fp32 rounding of l and of the
    logits (2^-19), times |V| < 5; a rounded P of key `pos` would be off by up to 2^-12."""
    rng = np.random.default_rng(pos)
    hd, T, H = (128, 300, 8) if form == "relpos" else (64, 1000 if "shared" in form else 256, 4)
    scale = 1.0 / 16
    q = np.zeros((1, H, T, hd), np.float16)
    k, v = np.zeros((1, H, T, hd), np.float16), randn_f16(rng, (1, H, T, hd))
    # q = (64, gap): k[0] = (1, 0) scores 4, k[pos] = (1, 1) scores 4 + gap / 16, the others (-7, 0) -28
    q[..., 0], k[..., 0] = 64.0, -7.0
    gap = np.linspace(8.2, 11.9, T) / np.log2(np.e) / scale
    q[..., 1] = gap.astype(np.float16)
    k[:, :, 0, 0], k[:, :, pos, 0], k[:, :, pos, 1] = 1.0, 1.0, 1.0
    kw = dict(scale=scale)
    if form == "relpos":
        kw.update(q_v=q, r=np.zeros((1, H, 2 * T - 1, hd), np.float16))
    got = gpu_op(b200, q, k, v, **kw)
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5
    w0 = np.exp(-q[0, :, :, 1].astype(np.float64) * scale)                       # key 0 against key `pos`
    v64 = v[0].astype(np.float64)
    want = (v64[:, pos][:, None] + w0[..., None] * v64[:, 0][:, None]) / (1.0 + w0)[..., None]
    assert np.abs(got[0].transpose(1, 0, 2) - want).max() <= 5 * (2.0 ** -20 + 2.0 ** -18)


@pytest.mark.parametrize("S,H,gqa,T", [(1, 6, 1, 500), (3, 8, 1, 500), (2, 12, 2, 700), (1, 20, 1, 1000), (5, 8, 4, 900)])
@pytest.mark.parametrize("form", ["plain", "causal", "lengths"])
@pytest.mark.parametrize("q_f32", [False, True])
def test_prefill_few_tiles_forms(b200, orc, S, H, gqa, T, form, q_f32):
    """head_dim 64 launches on both sides of each line of the choice between the four-CTA kernel, its shared tiles and the
    two-CTA kernel: 24 to 320 query tiles, F16 and F32 queries, grouped heads, causal, ragged lengths."""
    rng = np.random.default_rng(S * T + H)
    q, k, v = randn_f16(rng, (S, H, T, 64)), randn_f16(rng, (S, H // gqa, T, 64)), randn_f16(rng, (S, H // gqa, T, 64))
    if q_f32:
        q = q.astype(np.float32)
    kw = dict(scale=0.125)
    if form == "causal":
        kw.update(causal=True, n_past=0)
    if form == "lengths":
        kw.update(kv_len=np.linspace(1, T, S).astype(np.int32))
    rows = np.unique(np.linspace(0, T - 1, 60).astype(np.int32))
    got = gpu_op(b200, q, k, v, **kw)
    assert b200.lib().b200_last_kernel() == abi.KERNEL_PREFILL_TC5
    ref = orc.flash_attn_ext(q, k, v, rows=rows, **kw)
    assert_close(got[:, rows], ref[:, rows], f"S={S} H={H} gqa={gqa} T={T} {form}")
    assert b200.lib().b200_device_status() == 0


def test_workspace_out_of_memory_is_torchs_error(b200):
    """A workspace that the caching allocator cannot provide (here: beyond the process's share of the card) raises
    torch.OutOfMemoryError, on which servers free their caches and try again."""
    q = torch.randn(1, 20, 64, 64, device="cuda")
    k, v = (torch.randn(1, 20, 16384, 64, device="cuda") for _ in "kv")   # converted to F16: 84 MB of workspace
    out = torch.empty(1, 64, 20, 64, device="cuda")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (32 << 20)) / total)
        with pytest.raises(torch.OutOfMemoryError):
            b200.flash_attn_ext(q, k, v, scale=0.125, out=out)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert b200.flash_attn_ext(q, k, v, scale=0.125, out=out) is out
    torch.cuda.synchronize()


def test_workspace_of_a_launch_on_another_stream(b200, orc):
    """A call on an explicit stream takes its workspace from that stream's pool: a block that the current stream has freed but
    still reads (behind a delay) is not written, and the result does not depend on what the current stream allocates next."""
    rng = np.random.default_rng(5)
    q, k, v = (rng.standard_normal((1, 8, n, 64)).astype(np.float32) for n in (200, 9000, 9000))
    dq, dk, dv = (torch.from_numpy(x).cuda() for x in (q, k, v))
    out = torch.empty(1, 200, 8, 64, device="cuda")
    n = b200.workspace_bytes(dq, dk, dv, scale=0.125)
    assert n > 10 << 20
    side = torch.cuda.Stream()
    b200.flash_attn_ext(dq, dk, dv, scale=0.125, out=out)   # (the first launch of a kernel loads it, which waits for the device)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    x = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
    y = torch.empty_like(x)
    side.wait_stream(torch.cuda.current_stream())
    torch.cuda._sleep(200_000_000)      # about 0.1 s on the current stream; the launch below does not wait for it
    y.copy_(x)
    del x
    b200.flash_attn_ext(dq, dk, dv, scale=0.125, out=out, stream=side.cuda_stream)
    z = torch.full((n,), 9, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert bool((y == 7).all()) and bool((z == 9).all())
    assert_close(out.cpu().numpy(), orc.flash_attn_ext(q, k.astype(np.float16), v.astype(np.float16), scale=0.125), "launch on another stream")


@pytest.mark.parametrize("B,H,T", [(1, 20, 1500), (3, 20, 1500)])
def test_host_entry_point_result_over_its_query(b200, orc, B, H, T):
    """The result may take the place of the query: the heads of an entry, which lie apart in the query and side by side in the
    result, then have to be uploaded before any of them is written."""
    rng = np.random.default_rng(B)
    q, k, v = (randn_f16(rng, (B, H, T, 64)) for _ in "qkv")
    hq = torch.from_numpy(q.astype(np.float32)).pin_memory()
    hk, hv = torch.from_numpy(k).pin_memory(), torch.from_numpy(v).pin_memory()
    out = hq.view(B, T, H, 64)
    assert b200.flash_attn_ext_host(hq, hk, hv, scale=0.125, out=out) is out
    rows = np.arange(0, T, 37)
    assert_close(out.numpy()[:, rows], orc.flash_attn_ext(q, k, v, scale=0.125, rows=rows)[:, rows], "result in place of the query")


@pytest.mark.parametrize("kv_kind", ["f16", "q8_0"])
def test_head_dim_32_into_an_unaligned_result(b200, orc, kv_kind):
    """The result of head_dim 32 may start on any 4-byte boundary, decode steps without splits included."""
    rng = np.random.default_rng(1)
    q, k = randn_f16(rng, (2, 4, 3, 32)), rng.standard_normal((2, 2, 40, 32)).astype(np.float32)
    kw = dict(scale=32 ** -0.5)
    if kv_kind == "q8_0":
        kv, kw["kv_type"] = orc.quantize_q8_0(k), abi.Q8_0
    else:
        kv = k.astype(np.float16)
    out = torch.empty(2 * 3 * 4 * 32 + 1, device="cuda")[1:].view(2, 3, 4, 32)
    assert out.data_ptr() % 16 == 4
    dkv = torch.from_numpy(kv).cuda()
    b200.flash_attn_ext(torch.from_numpy(q).cuda(), dkv, dkv, out=out, **kw)
    torch.cuda.synchronize()
    assert b200.lib().b200_last_kernel() == abi.KERNEL_DECODE_SPLIT
    assert_close(out.cpu().numpy(), orc.flash_attn_ext(q, kv, kv, **kw), f"unaligned result, {kv_kind}")
