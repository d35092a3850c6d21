"""What a user of the framework has it do, as timed cases: quantized projections for one token, a decode batch and a
prefill chunk, the vocabulary projection, the KV write of a prefill chunk, attention over packed and f16 KV rows, and the
whole decode step.  Every case goes through the public entry points (`Kernels`, `QuantizedKvCache`, `DecodeModel`,
`CommandBatch`, `CudaGraph`).  Shapes are those of the synthetic E2B-like decoder (hidden 1536, FFN 6144, vocabulary
262144, 8 query heads and 1 KV head of 256, sliding window 512) and of the repository's tests.

A case is a dict of plain values; `kind` selects the entry point:

  matvec      m = 1, `layers` matrices of one shape against one vector each, one batch
  matmul      m >= 2, the same for a batch of rows
  vocab       f32 logits of m rows against one tall Q4_0 table
  kv_write    rows of K and V into a TurboQuant cache
  attend      one query position over a TurboQuant cache
  attend_b    one query position per lane over a pool of lanes
  prefill     a chunk of query rows over a TurboQuant cache
  attend_f16  one query position over f16 K and V
  step        one decode step of the whole model, recorded once as a graph and replayed
"""
import math

import torch

from __graft_entry__ import load_package

la = load_package()

ROW_BYTES = {"q4_0": lambda k: k // 32 * 18, "tq2_0": lambda k: k // 256 * 66}
_shared = []


def _program():
    """The context and kernel library that a program creates once."""
    if not _shared:
        torch.cuda.init()
        ctx = la.CudaContext.new(0)
        _shared.append((ctx, la.Kernels.new(ctx)))
    return _shared[0]


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # One Q4_0 projection for one token: the smallest call, where the launch and the host path count.
        {"name": "matvec_q4_0", "kind": "matvec", "fmt": "q4_0", "m": 1, "k": 1536, "n": 6144, "layers": 1},
        # The same TQ2_0 projection of every layer for a decode batch of 16: weights come from HBM each time.
        {"name": "matmul_tq2_0_m16", "kind": "matmul", "fmt": "tq2_0", "m": 16, "k": 1536, "n": 8192, "layers": 35},
        # FFN projection of a 256-row prefill chunk.
        {"name": "matmul_tq2_0_m256", "kind": "matmul", "fmt": "tq2_0", "m": 256, "k": 1536, "n": 6144, "layers": 1},
        # FFN down projection of a whole prompt with Q4_0 weights; prompts have odd lengths.
        {"name": "matmul_q4_0_m509", "kind": "matmul", "fmt": "q4_0", "m": 509, "k": 6144, "n": 1536, "layers": 1},
        # Logits of one sequence against the full vocabulary.
        {"name": "vocab_q4_0_m1", "kind": "vocab", "m": 1, "k": 1536, "n": 262144},
        # KV rows of one 256-row prefill chunk into a 4-bit cache.
        {"name": "kv_write_tq4_256", "kind": "kv_write", "bits": 4, "hd": 256, "n_kv": 1, "rows": 256, "position": 3841},
        # One long sequence, full-attention layer.
        {"name": "attend_tq2_32768", "kind": "attend", "bits": 2, "hd": 256, "n_q": 8, "n_kv": 1, "context": 32768},
        # A serving batch with ragged contexts and the most accurate codec.
        {"name": "attend_tq4_64_ragged", "kind": "attend_b", "bits": 4, "hd": 256, "n_q": 8, "n_kv": 1, "lanes": 64,
         "context": 8192, "ragged": True, "window": 0},
        # Attention of a 256-row prefill chunk that ends at 4096.
        {"name": "prefill_tq2_256x4096", "kind": "prefill", "bits": 2, "hd": 256, "n_q": 8, "n_kv": 1, "rows": 256,
         "context": 4096, "window": 0},
        # The cache without quantization, two KV heads.
        {"name": "attend_f16_8191", "kind": "attend_f16", "hd": 256, "n_q": 8, "n_kv": 2, "context": 8191},
        # The headline workloads: one decode step at batch 1 and at batch 64, context 8192.
        {"name": "step_b1", "kind": "step", "lanes": 1, "context": 8192, "layers": 35, "ring": 512, "ragged": False},
        {"name": "step_b64", "kind": "step", "lanes": 64, "context": 8192, "layers": 35, "ring": 512, "ragged": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matvec", "matmul", "matmul", "vocab", "kv_write", "attend", "attend_b", "prefill", "attend_f16", "step", "step"])
    if kind in ("matvec", "matmul"):
        m = 1 if kind == "matvec" else _log(rng, 2, 512)
        return {"kind": kind, "fmt": rng.choice(["q4_0", "tq2_0"]), "m": m, "k": 256 * _log(rng, 2, 32), "n": _log(rng, 512, 16384),
                "layers": rng.choice([1, 8, 35]) if m <= 64 else 1}
    if kind == "vocab":
        return {"kind": kind, "m": _log(rng, 1, 64), "k": rng.choice([1024, 1536, 2048]), "n": _log(rng, 32768, 262144)}
    hd, (n_q, n_kv) = rng.choice([128, 256, 256, 512]), rng.choice([(8, 1), (8, 1), (8, 2)])
    bits = rng.choice([2, 3, 4])
    if kind == "kv_write":
        return {"kind": kind, "bits": bits, "hd": hd, "n_kv": n_kv, "rows": _log(rng, 1, 4096), "position": rng.randrange(0, 4096)}
    if kind == "attend":
        return {"kind": kind, "bits": bits, "hd": hd, "n_q": n_q, "n_kv": n_kv, "context": _log(rng, 64, 131072)}
    if kind == "attend_b":
        return {"kind": kind, "bits": bits, "hd": hd, "n_q": n_q, "n_kv": n_kv, "lanes": _log(rng, 2, 64), "context": _log(rng, 64, 8192),
                "ragged": rng.random() < 0.7, "window": rng.choice([0, 0, 512])}
    if kind == "prefill":
        rows = _log(rng, 2, 256)
        return {"kind": kind, "bits": bits, "hd": min(hd, 256), "n_q": n_q, "n_kv": n_kv, "rows": rows, "context": rows + _log(rng, 64, 3840),
                "window": rng.choice([0, 512])}
    if kind == "attend_f16":
        return {"kind": kind, "hd": hd, "n_q": n_q, "n_kv": n_kv, "context": _log(rng, 64, 32768)}
    lanes = _log(rng, 1, 256)
    layers = rng.choice([n for n in (5, 10, 20, 35) if n == 5 or n * lanes <= 64 * 35])
    return {"kind": kind, "lanes": lanes, "context": _log(rng, 128, min(8192, 64 * 8192 * 35 // (lanes * layers))), "layers": layers,
            "ring": rng.choice([512, 1024]), "ragged": rng.random() < 0.5}


# ----------------------------------------------------------------- inputs --
class Owner:
    """Closes what the framework allocated once neither the state nor a tensor that views its memory needs it."""

    def __init__(self, ctx):
        self.ctx, self.closers, self.keep = ctx, [], []

    def __del__(self):
        try:
            self.ctx.synchronize()
            for close in reversed(self.closers):
                close()
        except TypeError:  # the interpreter is going down
            pass


class State:
    """A prepared case: what its program keeps between calls."""

    def __init__(self, seed):
        self.ctx, self.kernels = _program()
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.owner = Owner(self.ctx)
        self.pending, self.enqueue, self.graph, self.outputs = None, None, None, None

    def closes(self, close):
        self.owner.closers.append(close)

    def buf(self, t):
        b = la.CudaBuffer.wrap(self.ctx, t.data_ptr(), t.numel() * t.element_size())
        self.owner.keep.append(t)
        self.closes(b.free)
        return b

    def empty(self, shape, dtype):
        return torch.zeros(shape, dtype=dtype, device="cuda")

    def normal(self, *shape):
        return torch.randn(shape, generator=self.gen, dtype=torch.float16, device="cuda")

    def uniform(self, n, lo, hi):
        return torch.rand(n, generator=self.gen, device="cuda") * (hi - lo) + lo

    def ints(self, hi, n, dtype):
        return torch.randint(0, hi, (n,), generator=self.gen, device="cuda", dtype=dtype)

    def view(self, buf, shape, typestr):
        """A buffer that the framework owns, as a tensor."""
        return torch.as_tensor(_DeviceMemory(self.owner, buf, shape, typestr), device="cuda")

    def __del__(self):
        try:
            if self.pending is not None:
                self.pending.wait()
        except TypeError:  # the interpreter is going down
            pass


class _DeviceMemory:
    def __init__(self, owner, buf, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (buf.device_ptr, False), "version": 3}


def _q4_0(s, rows, cols):
    """GGUF Q4_0 blocks: f16 d ~ U[0.001, 0.02], 32 uniform 4-bit codes."""
    n = rows * (cols // 32)
    out = torch.empty((n, 18), dtype=torch.uint8, device="cuda")
    out[:, :2] = s.uniform(n, 0.001, 0.02).half().view(torch.uint8).view(n, 2)
    out[:, 2:] = s.ints(256, n * 16, torch.uint8).view(n, 16)
    return out


def _tq2_0(s, rows, cols):
    """GGUF TQ2_0 blocks: 256 uniform ternary codes, f16 d ~ U[0.005, 0.05]."""
    n = rows * (cols // 256)
    four = [a | b << 2 | c << 4 | d << 6 for a in range(3) for b in range(3) for c in range(3) for d in range(3)]
    four = torch.tensor(four, dtype=torch.uint8, device="cuda")
    out = torch.empty((n, 66), dtype=torch.uint8, device="cuda")
    out[:, :64] = four[s.ints(81, n * 64, torch.int32)].view(n, 64)
    out[:, 64:] = s.uniform(n, 0.005, 0.05).half().view(torch.uint8).view(n, 2)
    return out


WEIGHTS = {"q4_0": _q4_0, "tq2_0": _tq2_0}


def _codec(s, hd, bits):
    return (s.buf(torch.from_numpy(la.tq_levels(hd, bits)).cuda()), s.buf(torch.from_numpy(la.tq_signs(hd, la.TQ_SEED)).cuda()))


def _filled_rows(s, codes, norms, n_rows, n_kv, hd, bits, levels, signs):
    """Encodes n_rows normal rows into a pool."""
    for at in range(0, n_rows, 1 << 18):
        n = min(1 << 18, n_rows - at)
        x = s.normal(n, n_kv, hd)
        torch.cuda.synchronize()
        b = la.CommandBatch.new(s.ctx)
        src = la.CudaBuffer.wrap(s.ctx, x.data_ptr(), x.numel() * 2)
        s.kernels.encode_kv_turboquant_into(b, src, levels, signs, codes, norms, hd, n_kv, n, bits, at, 0)
        b.commit_and_wait()
        src.free()


def _filled_cache(s, case, n):
    cache = la.QuantizedKvCache(s.ctx, case["n_kv"], case["hd"], n, bits=case["bits"])
    s.closes(cache.close)
    p = cache.buffers()
    for codes, norms in (("keys_q", "key_norms"), ("values_q", "value_norms")):
        _filled_rows(s, p[codes], p[norms], n, case["n_kv"], case["hd"], case["bits"], p["levels"], p["signs"])
    return cache


def _positions(s, case):
    """The newest position of each lane: all the same, or lognormal around a quarter of the longest."""
    lanes, most = case["lanes"], case["context"]
    if not case["ragged"]:
        return torch.full((lanes,), most - 1, dtype=torch.int32, device="cuda")
    x = torch.randn(lanes, generator=s.gen, device="cuda").exp() * (most / 4)
    return x.round().clamp(min(16, most), most).int() - 1


def prepare(case, seed):
    s = State(seed)
    PREPARE[case["kind"]](s, case)
    torch.cuda.synchronize()
    return s


def _prepare_matmul(s, case):
    m, k, n = case["m"], case["k"], case["n"]
    x = s.buf(s.normal(m, k))
    ws = [s.buf(WEIGHTS[case["fmt"]](s, n, k)) for _ in range(case["layers"])]
    outs = [s.empty((m, n), torch.float16) for _ in ws]
    pairs = list(zip(ws, [s.buf(o) for o in outs]))
    if m == 1:
        op = getattr(s.kernels, "matvec_%s_into" % case["fmt"])
        s.enqueue = lambda b: [op(b, w, x, o, n, k) for w, o in pairs]
    else:
        op = getattr(s.kernels, "matmul_nt_%s_into" % case["fmt"])
        s.enqueue = lambda b: [op(b, x, w, o, m, k, n) for w, o in pairs]
    s.outputs = outs


def _prepare_vocab(s, case):
    kernels = s.kernels
    m, k, n = case["m"], case["k"], case["n"]
    x, w, out = s.buf(s.normal(m, k)), s.buf(_q4_0(s, n, k)), s.empty((m, n), torch.float32)
    o = s.buf(out)
    if m == 1:
        s.enqueue = lambda b: kernels.matvec_q4_0_f32out_into(b, w, x, o, n, k)
    else:
        s.enqueue = lambda b: kernels.matmul_nt_q4_0_f32out_into(b, x, w, o, m, k, n)
    s.outputs = out


def _prepare_kv_write(s, case):
    kernels = s.kernels
    rows, at, hd, n_kv = case["rows"], case["position"], case["hd"], case["n_kv"]
    k, v = s.buf(s.normal(rows, n_kv, hd)), s.buf(s.normal(rows, n_kv, hd))
    n = at + rows
    cache = la.QuantizedKvCache(s.ctx, n_kv, hd, n, bits=case["bits"])
    s.closes(cache.close)
    s.enqueue = lambda b: cache.write_kv_gpu_into(b, kernels, k, v, at, rows)
    p, cb = cache.buffers(), cache.code_bytes()
    s.outputs = {x: s.view(p[x], (n, n_kv, cb), "|u1") for x in ("keys_q", "values_q")}
    s.outputs.update({x: s.view(p[x], (n, n_kv), "<i2") for x in ("key_norms", "value_norms")})  # bit patterns of the f16 norms


def _prepare_attend(s, case):
    kernels = s.kernels
    n, n_q, hd = case["context"], case["n_q"], case["hd"]
    cache, q, out = _filled_cache(s, case, n), s.buf(s.normal(n_q, hd)), s.empty((n_q, hd), torch.float16)
    o, scale = s.buf(out), hd ** -0.5
    s.enqueue = lambda b: cache.fused_attention_into(b, kernels, q, o, n, n - 1, n_q, 0, scale)
    s.outputs = out


def _prepare_prefill(s, case):
    kernels = s.kernels
    n, rows, n_q, hd = case["context"], case["rows"], case["n_q"], case["hd"]
    cache, q, out = _filled_cache(s, case, n), s.buf(s.normal(rows, n_q, hd)), s.empty((rows, n_q, hd), torch.float16)
    o, scale = s.buf(out), hd ** -0.5
    s.enqueue = lambda b: cache.fused_attention_batch_into(b, kernels, q, o, n, n - rows, rows, n_q, case["window"], scale)
    s.outputs = out


def _prepare_attend_b(s, case):
    kernels = s.kernels
    lanes, n, n_q, n_kv, hd, bits = (case[x] for x in ("lanes", "context", "n_q", "n_kv", "hd", "bits"))
    levels, signs = _codec(s, hd, bits)
    cb = la.tq_code_bytes(hd, bits)
    pools = []
    for _ in range(2):
        codes, norms = s.buf(s.empty((lanes * n * n_kv * cb,), torch.uint8)), s.buf(s.empty((lanes * n * n_kv,), torch.float16))
        _filled_rows(s, codes, norms, lanes * n, n_kv, hd, bits, levels, signs)
        pools += [codes, norms]
    q, out, pos = s.buf(s.normal(lanes, n_q, hd)), s.empty((lanes, n_q, hd), torch.float16), s.buf(_positions(s, case))
    o, scale = s.buf(out), hd ** -0.5
    s.enqueue = lambda b: kernels.tq_attention_batched_into(b, q, *pools, levels, signs, o, pos, hd, n, n_q, n_kv, case["window"],
                                                              bits, lanes, 0, scale)
    s.outputs = out


def _prepare_attend_f16(s, case):
    ctx, kernels = s.ctx, s.kernels
    n, n_q, n_kv, hd = case["context"], case["n_q"], case["n_kv"], case["hd"]
    # the entry point's softmax scale is 1: queries carry it, as after q-norm
    q, out = s.buf((s.normal(n_q, hd) * hd ** -0.5)), s.empty((n_q, hd), torch.float16)
    k, v, o = s.buf(s.normal(n, n_kv, hd)), s.buf(s.normal(n, n_kv, hd)), s.buf(out)
    s.enqueue = lambda b: kernels.flash_decoding_into(ctx, b, q, k, v, o, hd, n, n - 1, n_q, n_kv)
    s.outputs = out


def _prepare_step(s, case):
    lanes, n, layers = case["lanes"], case["context"], case["layers"]
    cfg = la.e2b_like_config(max_lanes=lanes, max_context=n + 64, n_layers=layers, swa_ring=case["ring"])
    model = la.DecodeModel(s.ctx, s.kernels, cfg)
    s.closes(model.close)
    near_one = lambda dim: s.buf((1 + 0.05 * s.normal(dim).float()).half())
    levels, signs = _codec(s, cfg.head_dim, cfg.kv_bits)
    pools = []
    for i in range(layers):
        t = {name: s.buf(_tq2_0(s, r, c)) for name, (r, c) in la.model.layer_shapes(cfg).items()}
        t.update({name: near_one(cfg.hidden) for name in ("attn_norm", "post_attn_norm", "ffn_norm", "post_ffn_norm")})
        t.update({name: near_one(cfg.head_dim) for name in ("q_norm", "k_norm")})
        torch.cuda.synchronize()
        model.set_layer(i, t)
        kv = model.kv_buffers(i)
        for x in ("k", "v"):
            _filled_rows(s, kv[x + "_codes"], kv[x + "_norms"], lanes * kv["lane_rows"], cfg.n_kv_heads, cfg.head_dim, cfg.kv_bits,
                         levels, signs)
        pools.append(kv)
    model.set_embedding(s.buf(_q4_0(s, cfg.vocab, cfg.hidden)), near_one(cfg.hidden))
    tokens, positions = s.buf(s.ints(cfg.vocab, lanes, torch.int32)), s.buf(_positions(s, case))
    chosen = s.buf(s.empty((lanes,), torch.int32))
    torch.cuda.synchronize()
    b = la.CommandBatch.new(s.ctx)  # once as it is: scratch memory cannot grow while a graph is recorded
    model.decode_batch_step_into(b, tokens, positions, lanes, True, chosen)
    b.commit_and_wait()
    b = la.CommandBatch.capture(s.ctx)
    model.decode_batch_step_into(b, tokens, positions, lanes, True, chosen)
    s.graph = b.end_capture()
    s.closes(s.graph.destroy)
    # Logits, final hidden rows and the KV rows of the deepest sliding and full layers.  The chosen tokens follow from the
    # logits; two that nearly tie may change places with the rounding, so they are not compared.
    s.outputs = {"logits": s.view(model.logits_buffer(), (lanes, cfg.vocab), "<f4"),
                 "hidden": s.view(model.hidden_buffer(), (lanes, cfg.hidden), "<f2")}
    cb = la.tq_code_bytes(cfg.head_dim, cfg.kv_bits)
    for i in (layers - 2, layers - 1):
        rows = lanes * pools[i]["lane_rows"]
        for x in ("k", "v"):
            s.outputs["%s_codes.%d" % (x, i)] = s.view(pools[i][x + "_codes"], (rows, cb), "|u1")
            s.outputs["%s_norms.%d" % (x, i)] = s.view(pools[i][x + "_norms"], (rows,), "<f2")


PREPARE = {"matvec": _prepare_matmul, "matmul": _prepare_matmul, "vocab": _prepare_vocab, "kv_write": _prepare_kv_write,
           "attend": _prepare_attend, "attend_b": _prepare_attend_b, "prefill": _prepare_prefill, "attend_f16": _prepare_attend_f16,
           "step": _prepare_step}


def run(s):
    if s.graph is not None:
        s.graph.launch()
        return s.outputs
    if s.pending is not None:  # this state's buffers are in use until its last pass is done
        s.pending.wait()
    b = la.CommandBatch.new(s.ctx)
    s.enqueue(b)
    s.pending = b.commit_async()
    return s.outputs


# ------------------------------------------------------------------- work --
def _mean_context(case):
    """Mean keys per lane: a lognormal(0, 1) variable over 4, clipped to 1, has mean 0.351."""
    return case["context"] * (0.351 if case.get("ragged") else 1.0)


def work(case):
    kind = case["kind"]
    if kind in ("matvec", "matmul", "vocab"):
        m, k, n, layers = case["m"], case["k"], case["n"], case.get("layers", 1)
        out = 4 if kind == "vocab" else 2
        return {"bytes": m * k * 2 + layers * (n * ROW_BYTES[case.get("fmt", "q4_0")](k) + m * n * out), "flops": layers * 2.0 * m * k * n}
    if kind == "step":
        lanes, layers = case["lanes"], case["layers"]
        weights = layers * sum(r * ROW_BYTES["tq2_0"](c) for r, c in la.model.layer_shapes(la.e2b_like_config()).values())
        table = 262144 * ROW_BYTES["q4_0"](1536)
        full = layers // 5
        near = min(512.0, _mean_context(case))
        keys = lanes * (full * _mean_context(case) + (layers - full) * near)
        macs = lanes * (weights * 256 / 66 + 262144 * 1536) + keys * 8 * 256 * 2
        return {"bytes": weights + table + keys * 132 + lanes * 262144 * 4, "flops": 2.0 * macs}
    hd, n_kv = case["hd"], case["n_kv"]
    row = hd * case["bits"] // 8 + 2 if "bits" in case else 2 * hd
    if kind == "kv_write":
        n = 2 * case["rows"] * n_kv
        return {"bytes": n * (2 * hd + row), "flops": n * hd * (math.log2(hd) + 6)}
    n_q, lanes, keys = case["n_q"], case.get("lanes", 1), _mean_context(case)
    rows = case.get("rows", 1)
    window = case.get("window") or keys
    seen = min(keys, window) if rows == 1 else min(keys - (rows - 1) / 2, window)  # keys per query row
    read = min(keys, window + rows - 1)
    return {"bytes": lanes * (read * n_kv * 2 * row + rows * n_q * hd * 4), "flops": 4.0 * lanes * rows * n_q * seen * hd}


def tolerance(case):
    if case["kind"] == "kv_write":
        return "exact"
    if case["kind"] == "vocab":  # f32 sums of exact products
        return {"rel": 2e-5, "max": 1e-3}
    if case["kind"] in ("matvec", "matmul"):  # f32 sums, stored as f16: two roundings that fall on either side
        return {"rel": 5e-4, "max": 2e-3}
    if case["kind"] == "step":  # f16 between the operations of 35 layers, KV codes that flip at a level's edge: about 5e-3
        return {"rel": 2e-2, "differ": 1e-2}
    return {"rel": 2e-3, "max": 2e-2}  # attention: f32 softmax over sums of f16 products, stored as f16
