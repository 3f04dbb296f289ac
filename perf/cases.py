"""The work that users of this library have it do, as measurable cases: the attention of Whisper decode steps and
encoders, of LLM decoders over their KV caches (decode steps and causal prefill), of FastConformer encoders with
relative positions, and the host-buffer round trip.

A case is a dict of plain values; `prepare` makes what a runtime holds before the call, `run` is one pass through the
public entry points, `work` is what the pass cannot do without and `tolerance` what another correct implementation at
the same precision may differ by.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

import crispasr_b200 as b200
from crispasr_b200 import abi

ENC_FRAMES = 1500      # frames of a 30 s Whisper window
POOL_CELLS = 3584      # cells of whisper's unified beam pool
TYPE_BYTES = {"f16": 2, "f32": 4}
TORCH_TYPE = {"f16": torch.float16, "f32": torch.float32}


def listed():
    return [
        # One decode step of Whisper base.en for a single 30 s window, beam 5: per layer the self-attention over the
        # cell pool with the dense membership mask, then the cross-attention over the encoder's K/V.  The smallest
        # calls there are: latency and launches.
        dict(name="whisper_base_step_1", kind="whisper_step", layers=6, heads=8, segments=1, beams=5, tokens=48, form="dense"),
        # The same step of Whisper large-v3 with the beams' cells as one shared index list: an interactive transcription.
        dict(name="whisper_large_step_1", kind="whisper_step", layers=32, heads=20, segments=1, beams=5, tokens=224, form="union"),
        # A transcription server: 32 windows step together (four of the 32 layers, so that the state stays small).
        dict(name="whisper_large_step_32", kind="whisper_step", layers=4, heads=20, segments=32, beams=5, tokens=448, form="union"),
        # One token of 8 resident streams of a Voxtral-mini-3B-style decoder over a Q8_0 cache: quantise-on-append and
        # attention in each of 30 layers, ragged lengths read on the device.
        dict(name="llm_step_q8_8", kind="llm_step", layers=30, heads=32, kv_heads=8, streams=8, ctx=535, kv="q8_0", q="f32"),
        # The same decoder over an F16 cache at 32 streams: a batch server.
        dict(name="llm_step_f16_32", kind="llm_step", layers=30, heads=32, kv_heads=8, streams=32, ctx=663, kv="f16", q="f16"),
        # Its prefill: 375 audio and 32 text tokens of 8 streams enter the Q8_0 cache and attend causally (one layer).
        dict(name="llm_prefill_q8_8", kind="llm_prefill", heads=32, kv_heads=8, streams=8, tokens=407, kv="q8_0", q="f32"),
        # Whisper large-v3 encoder, one layer over a batch of 64 windows: the benchmark's own workload.
        dict(name="whisper_large_encoder_64", kind="encoder", heads=20, segments=64, frames=1500, pad=0, q="f16", kv="f16"),
        # Whisper base.en encoder, one window, the operands as the runtime hands them over: an F32 query, token-major
        # K/V views padded to 1536 rows.
        dict(name="whisper_base_encoder_1", kind="encoder", heads=8, segments=1, frames=1500, pad=36, q="f32", kv="f16"),
        # Voxtral audio encoder, four windows: F32 query, keys and values.
        dict(name="voxtral_encoder_f32_4", kind="encoder", heads=20, segments=4, frames=1500, pad=0, q="f32", kv="f32"),
        # FastConformer encoder (Parakeet / Canary dimensions) over a batch of short utterances of different lengths
        # (at most 11 s), F32 strided views of the fused projection, untied position biases folded into the call.
        dict(name="fastconformer_short_8", kind="relpos", heads=8, utterances=8, frames=138, ragged=True, qkv="f32", masked=False),
        # The same encoder over two 10-minute recordings (7500 frames each).
        dict(name="fastconformer_long_2", kind="relpos", heads=8, utterances=2, frames=7500, ragged=False, qkv="f16", masked=False),
        # The operator for a runtime that keeps its tensors in (pinned) host memory: four windows of the large encoder.
        dict(name="host_encoder_4", kind="host_encoder", heads=20, segments=4, frames=1500, q="f16", kv="f16"),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, evenly over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    while True:
        kind = rng.choice(("whisper_step", "whisper_step", "llm_step", "llm_step", "llm_prefill", "encoder", "encoder", "relpos",
                           "relpos", "host_encoder"))
        if kind == "whisper_step":
            c = dict(kind=kind, layers=_spread(rng, 4, 32), heads=rng.choice((6, 8, 12, 16, 20)), segments=_spread(rng, 1, 32),
                     beams=rng.randint(1, 5), tokens=_spread(rng, 4, 448), form=rng.choice(("dense", "union", "index")))
        elif kind == "llm_step":
            heads, kv_heads = rng.choice(((32, 8), (16, 8), (16, 4), (8, 8)))
            c = dict(kind=kind, layers=_spread(rng, 8, 30), heads=heads, kv_heads=kv_heads, streams=_spread(rng, 1, 64),
                     ctx=_spread(rng, 60, 1300), kv=rng.choice(("q8_0", "f16")), q=rng.choice(("f32", "f16")))
        elif kind == "llm_prefill":
            heads, kv_heads = rng.choice(((32, 8), (16, 8), (16, 4), (8, 8)))
            c = dict(kind=kind, heads=heads, kv_heads=kv_heads, streams=_spread(rng, 1, 16), tokens=_spread(rng, 24, 1600),
                     kv=rng.choice(("q8_0", "f16")), q=rng.choice(("f32", "f16")))
        elif kind == "encoder":
            c = dict(kind=kind, heads=rng.choice((6, 8, 12, 16, 20)), segments=_spread(rng, 1, 64), frames=_spread(rng, 150, 1500),
                     pad=rng.choice((0, 0, 36)), q=rng.choice(("f32", "f16")), kv=rng.choice(("f16", "f16", "f32")))
        elif kind == "relpos":
            c = dict(kind=kind, heads=8, utterances=_spread(rng, 1, 16), frames=_spread(rng, 30, 7500), ragged=rng.random() < 0.5,
                     qkv=rng.choice(("f32", "f16")), masked=rng.random() < 0.2)
        else:
            c = dict(kind=kind, heads=rng.choice((6, 8, 12, 16, 20)), segments=_spread(rng, 1, 4), frames=_spread(rng, 150, 1500),
                     q=rng.choice(("f32", "f16")), kv="f16")
        w = work(c)
        if w["flops"] <= 740e9 and w["bytes"] <= (60e6 if kind == "host_encoder" else 2.7e9):
            return c


# ---- lengths ------------------------------------------------------------------------------------------------------

def _stream_lengths(c):
    """Keys of each resident stream after this step's append: they joined at different times."""
    return [c["ctx"] - (i * 37) % max(1, c["ctx"] // 3) for i in range(c["streams"])]


def _utterance_lengths(c):
    T, n = c["frames"], c["utterances"]
    return [T - (i * T // (2 * n) if c["ragged"] else 0) for i in range(n)]


def _live_cells(c):
    """(shared prefix, private suffix per beam) of a beam search at `tokens` positions: half of them shared."""
    prefix = c["tokens"] // 2
    return prefix, c["tokens"] - prefix


# ---- what a pass cannot do without ----------------------------------------------------------------------------------

def work(c):
    kind = c["kind"]
    if kind == "whisper_step":
        prefix, suffix = _live_cells(c)
        per_layer_rows = prefix + c["beams"] * suffix + ENC_FRAMES
        kv = 2 * per_layer_rows * 64 * 2
        qo = 2 * c["beams"] * 64 * (2 + 4)
        n = c["layers"] * c["heads"] * c["segments"]
        return {"bytes": n * (kv + qo), "flops": n * 4.0 * c["beams"] * 64 * per_layer_rows}
    if kind == "llm_step":
        row = 256 if c["kv"] == "f16" else 136
        keys = sum(_stream_lengths(c))
        kv = c["kv_heads"] * row * 2 * keys
        new = c["streams"] * c["kv_heads"] * 2 * 128 * 4
        qo = c["streams"] * c["heads"] * 128 * (TYPE_BYTES[c["q"]] + 4)
        return {"bytes": c["layers"] * (kv + new + qo), "flops": c["layers"] * 4.0 * c["heads"] * 128 * keys}
    if kind == "llm_prefill":
        row = 256 if c["kv"] == "f16" else 136
        n, T = c["streams"], c["tokens"]
        # the F32 rows in, the cache rows out (and in again), the query in, the output out
        nbytes = n * T * (c["kv_heads"] * 2 * (128 * 4 + 2 * row) + c["heads"] * 128 * (TYPE_BYTES[c["q"]] + 4))
        return {"bytes": nbytes, "flops": n * 2.0 * T * (T + 1) * 128 * c["heads"]}
    if kind in ("encoder", "host_encoder"):
        n, T, Lk = c["segments"] * c["heads"], c["frames"], c["frames"] + c.get("pad", 0)
        nbytes = n * 64 * (T * (TYPE_BYTES[c["q"]] + 4) + 2 * Lk * TYPE_BYTES[c["kv"]])
        return {"bytes": nbytes, "flops": n * 4.0 * T * Lk * 64}
    lens, H, es = _utterance_lengths(c), c["heads"], TYPE_BYTES[c["qkv"]]
    nbytes = sum(lens) * H * 128 * (3 * es + 4) + (2 * c["frames"] - 1) * H * 128 * 2
    if c["masked"]:
        nbytes += 2 * c["frames"] ** 2
    # scores, bias products (one per score) and the weighted sum
    return {"bytes": nbytes, "flops": sum(6.0 * n * n * 128 * H for n in lens)}


def tolerance(c):
    # F16 tensor-core operands (queries, keys, probabilities; rounding 2^-11 each) under fp32 softmax and accumulation;
    # cache rows are the same bits
    return {"rel": 1e-3, "max": 2e-2, "differ": 0.0}


# ---- inputs ---------------------------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, shape, dtype, scale=1.0):
    x = torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)
    return (x * scale if scale != 1.0 else x).to(dtype)


def _token_major(g, batch, rows, heads, hd, dtype, scale=1.0, pad=0):
    """(B, H, rows + pad, hd) view of a token-major buffer with interleaved heads; the padding rows are zero."""
    buf = torch.zeros((batch, rows + pad, heads, hd), dtype=dtype, device="cuda")
    buf[:, :rows] = _randn(g, (batch, rows, heads, hd), dtype, scale)
    return buf.permute(0, 2, 1, 3)


class _DeviceBytes:
    """Device memory of a KV cache described to torch; keeps the cache alive as long as the tensor."""

    def __init__(self, cache, ptr, shape, typestr, strides=None):
        self.cache = cache
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=tuple(shape), typestr=typestr, strides=strides, version=3)


def _slab_view(cache, t, dtype):
    """(streams, kv heads, rows, row) torch view of a cache descriptor."""
    if dtype == "q8_0":
        last, es, typestr = t.ne[0] // 32 * 34, 1, "|u1"
    else:
        last, es, typestr = t.ne[0], 2, "<f2"
    return torch.as_tensor(_DeviceBytes(cache, t.data, (t.ne[3], t.ne[2], t.ne[1], last), typestr, (t.nb[3], t.nb[2], t.nb[1], es)), device="cuda")


def prepare(case, seed):
    c, g = dict(case), _gen(seed)
    kind = c["kind"]
    if kind == "whisper_step":
        return _prepare_whisper_step(c, g, seed)
    if kind in ("llm_step", "llm_prefill"):
        return _prepare_llm(c, g)
    if kind in ("encoder", "host_encoder"):
        q = _randn(g, (c["segments"], c["frames"], c["heads"], 64), TORCH_TYPE[c["q"]]).permute(0, 2, 1, 3)
        k, v = (_token_major(g, c["segments"], c["frames"], c["heads"], 64, TORCH_TYPE[c["kv"]], pad=c.get("pad", 0)) for _ in "kv")
        if kind == "encoder" and not c["pad"]:   # without padding the runtimes hand over head-major tensors
            q, k, v = q.contiguous(), k.contiguous(), v.contiguous()
        st = dict(case=c, q=q, k=k, v=v)
        if kind == "host_encoder":
            for name in "qkv":
                x = st[name].contiguous()
                st[name] = torch.empty(x.shape, dtype=x.dtype, pin_memory=True).copy_(x)
            st["out"] = torch.empty((c["segments"], c["frames"], c["heads"], 64), dtype=torch.float32, pin_memory=True)
        return st
    return _prepare_relpos(c, g)


def _prepare_whisper_step(c, g, seed):
    S, H, beams, layers = c["segments"], c["heads"], c["beams"], c["layers"]
    prefix, suffix = _live_cells(c)
    live = prefix + beams * suffix
    n_cells = -(-live // 256) * 256 if c["form"] == "dense" else POOL_CELLS
    # the pool as a running beam search leaves it: a shared prefix and private cells, scattered
    prng = np.random.default_rng(seed)
    slots = prng.permutation(n_cells)[:live]
    pos, bits = np.full(n_cells, -1, np.int32), np.zeros(n_cells, np.uint32)
    pos[slots[:prefix]], bits[slots[:prefix]] = np.arange(prefix), (1 << beams) - 1
    for j in range(beams):
        own = slots[prefix + j * suffix:prefix + (j + 1) * suffix]
        pos[own], bits[own] = prefix + np.arange(suffix), 1 << j
    tok_seq, tok_pos = np.arange(beams, dtype=np.int32), np.full(beams, prefix + suffix - 1, np.int32)
    L, kw, mask = b200.lib(), dict(scale=1.0), None
    if c["form"] == "dense":
        seen = ((bits[None, :] >> tok_seq[:, None].astype(np.uint32)) & 1).astype(bool) & (pos[None, :] <= tok_pos[:, None])
        mask = torch.from_numpy(np.where(seen, 0.0, -np.inf).astype(np.float16)[None, None]).cuda()
    elif c["form"] == "union":
        stride = -(-live // 64) * 64
        idx, n, m = np.zeros(stride, np.int32), np.zeros(1, np.int32), np.zeros((beams, stride), np.uint16)
        if L.b200_beam_cells_to_union(pos.ctypes.data, bits.ctypes.data, n_cells, tok_seq.ctypes.data, tok_pos.ctypes.data, beams,
                                      idx.ctypes.data, stride, n.ctypes.data, m.ctypes.data):
            raise RuntimeError("b200_beam_cells_to_union")
        mask = torch.from_numpy(m.view(np.float16)[None, None]).cuda()
        kw.update(kv_index=torch.from_numpy(np.tile(idx[None], (S, 1))).cuda(), kv_len=torch.from_numpy(np.tile(n, S)).cuda())
    else:
        stride = prefix + suffix
        idx, n = np.zeros((beams, stride), np.int32), np.zeros(beams, np.int32)
        if L.b200_beam_cells_to_index(pos.ctypes.data, bits.ctypes.data, n_cells, tok_seq.ctypes.data, tok_pos.ctypes.data, beams,
                                      idx.ctypes.data, stride, n.ctypes.data):
            raise RuntimeError("b200_beam_cells_to_index")
        kw.update(kv_index=torch.from_numpy(np.tile(idx, (S, 1))).cuda(), kv_len=torch.from_numpy(np.tile(n, S)).cuda())
    per_layer = []
    for _ in range(layers):
        # queries of the step's tokens, token-major as the projection leaves them; the self-attention's are pre-scaled
        q = _randn(g, (S, beams, H, 64), torch.float16, 0.5 * 64 ** -0.25)
        qx = _randn(g, (S, beams, H, 64), torch.float16, 0.5).permute(0, 2, 1, 3)
        # with one list per beam the beams are batch entries that share their segment's pool
        q = q.reshape(S * beams, 1, H, 64).permute(0, 2, 1, 3) if c["form"] == "index" else q.permute(0, 2, 1, 3)
        k, v = (_token_major(g, S, n_cells, H, 64, torch.float16, 0.5) for _ in "kv")
        xk, xv = (_token_major(g, S, ENC_FRAMES, H, 64, torch.float16, 0.5) for _ in "kv")
        per_layer.append((q, k, v, qx, xk, xv))
    return dict(case=c, layers=per_layer, mask=mask, kw=kw)


def _prepare_llm(c, g):
    step = c["kind"] == "llm_step"
    layers, S, H, Hkv = c.get("layers", 1), c["streams"], c["heads"], c["kv_heads"]
    lens = _stream_lengths(c) if step else [c["tokens"]] * S
    n_new = 1 if step else c["tokens"]
    cache = b200.KvCache(abi.Q8_0 if c["kv"] == "q8_0" else abi.F16, 128, Hkv, layers, max(lens), S)
    kv_len = torch.tensor(lens, dtype=torch.int32, device="cuda")
    st = dict(case=c, cache=cache, kv_len=kv_len, pos=kv_len - 1, q=[], new=[], views=[])
    for i in range(layers):
        if step:   # the rows of the earlier tokens
            cache.append(i, *(_randn(g, (S, Hkv, max(lens), 128), torch.float32) for _ in "kv"), pos0=0)
        st["views"].append([_slab_view(cache, t, c["kv"]) for t in cache.view(i, max(lens))])
        # token-major rows of the projections
        st["q"].append(_randn(g, (S, n_new, H, 128), TORCH_TYPE[c["q"]]).permute(0, 2, 1, 3))
        st["new"].append([_randn(g, (S, n_new, Hkv, 128), torch.float32).permute(0, 2, 1, 3) for _ in "kv"])
    # the whole cache, slab after slab, as the state that a pass updates
    n = cache.nbytes
    first = cache.view(0, 1)[0].data
    st["rows"] = torch.as_tensor(_DeviceBytes(cache, first, (n,), "|u1") if c["kv"] == "q8_0" else _DeviceBytes(cache, first, (n // 2,), "<f2"),
                                 device="cuda")
    return st


def _prepare_relpos(c, g):
    B, T, H, hd = c["utterances"], c["frames"], c["heads"], 128
    dt, d = TORCH_TYPE[c["qkv"]], H * hd
    qkv = _randn(g, (B, T, 3, H, hd), dt)             # the fused projection's rows
    q, k, v = (qkv[:, :, i].permute(0, 2, 1, 3) for i in range(3))
    bias_u, bias_v = (_randn(g, (H, hd), torch.float32, 0.02) for _ in "uv")
    w_pos = _randn(g, (d, d), torch.float32, d ** -0.5)
    r = torch.empty((1, H, 2 * T - 1, hd), dtype=torch.float16, device="cuda")
    tw = abi.from_torch(w_pos)
    rc = b200.lib().b200_relpos_table(C.byref(tw), H, T, r.data_ptr(), r.numel() * 2, torch.cuda.current_stream().cuda_stream)
    if rc:
        raise RuntimeError("b200_relpos_table: %d" % rc)
    kw = dict(scale=hd ** -0.5, r=r, pos_bias_u=bias_u, pos_bias_v=bias_v)
    if c["ragged"]:
        lens = torch.tensor(_utterance_lengths(c), dtype=torch.int32, device="cuda")
        kw.update(q_len=lens, kv_len=lens)
    mask = None
    if c["masked"]:   # limited context: each frame sees a window of frames around itself
        i = torch.arange(T, device="cuda")
        near = (i[None, :] - i[:, None]).abs() <= max(8, T // 4)
        mask = torch.where(near, 0.0, float("-inf")).to(torch.float16)[None, None]
    return dict(case=c, q=q, k=k, v=v, mask=mask, kw=kw)


# ---- one pass -------------------------------------------------------------------------------------------------------

def run(st):
    c = st["case"]
    kind = c["kind"]
    if kind == "whisper_step":
        outs = []
        for q, k, v, qx, xk, xv in st["layers"]:
            outs.append(b200.flash_attn_ext(q, k, v, st["mask"], **st["kw"]))
            outs.append(b200.flash_attn_ext(qx, xk, xv, scale=64 ** -0.25))
        return outs
    if kind == "llm_step":
        outs = []
        kv_type = abi.Q8_0 if c["kv"] == "q8_0" else None
        for i in range(c["layers"]):
            st["cache"].append(i, *st["new"][i], pos=st["pos"])
            outs.append(b200.flash_attn_ext(st["q"][i], *st["views"][i], scale=128 ** -0.5, kv_type=kv_type, kv_len=st["kv_len"]))
        return outs + [st["rows"]]
    if kind == "llm_prefill":
        kv_type = abi.Q8_0 if c["kv"] == "q8_0" else None
        st["cache"].append(0, *st["new"][0], pos0=0)
        out = b200.flash_attn_ext(st["q"][0], *st["views"][0], scale=128 ** -0.5, kv_type=kv_type, causal=True)
        return [out, st["rows"]]
    if kind == "encoder":
        return b200.flash_attn_ext(st["q"], st["k"], st["v"], scale=0.125)
    if kind == "host_encoder":
        return b200.flash_attn_ext_host(st["q"], st["k"], st["v"], scale=0.125, out=st["out"])
    return b200.flash_attn_ext(st["q"], st["k"], st["v"], st["mask"], **st["kw"])
