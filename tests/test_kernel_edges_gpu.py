"""The tensor-core kernels at the sizes where their tiling can go wrong: tile edges, remainders, the smallest and the
largest of each dispatch range, against the CPU oracle."""
import time

import numpy as np
import pytest

from gpu_util import Guarded, rel_close
from test_attention_gpu import Cache, f16_case
from test_matvec_gpu import device_status_ok, run_matmul
from test_turboquant_gpu import gpu_encode

pytestmark = pytest.mark.gpu


# m <= 16: one 8- or 16-row tile; K in 32- (Q4_0) or 256-wide (TQ2_0) blocks, uneven over the warps; ragged last rows of W.
# m > 64, and Q4_0 from 17: 128-row weight tiles, batch tiles of 64 / 128 columns, K splits with a remainder.
@pytest.mark.parametrize("fmt,m,k,n", [
    ("q4_0", 1, 32, 1), ("q4_0", 8, 96, 65), ("q4_0", 9, 1536, 129), ("q4_0", 16, 2080, 63), ("q4_0", 16, 6144, 1537), ("q4_0", 11, 1792, 14213),
    ("tq2_0", 9, 256, 127), ("tq2_0", 16, 768, 8193), ("tq2_0", 13, 2048, 33), ("tq2_0", 16, 2304, 6000),
    ("tq2_0", 16, 6144, 1537),
    ("q4_0", 17, 96, 127), ("q4_0", 64, 1568, 129), ("q4_0", 65, 32, 1), ("q4_0", 129, 2080, 130), ("q4_0", 257, 1536, 300),
    ("tq2_0", 65, 256, 127), ("tq2_0", 128, 1536, 129), ("tq2_0", 129, 6144, 260), ("tq2_0", 300, 768, 1)])
def test_quantised_matmul_at_tile_edges(la, orc, ctx, kernels, fmt, m, k, n):
    raw = (la.synth.q4_0_weights if fmt == "q4_0" else la.synth.tq2_0_weights)(n, k, 31)
    a = la.synth.normal_f16((m, k), 32)
    want = orc.matmul_nt(orc.Q4_0 if fmt == "q4_0" else orc.TQ2_0, a, raw, m, k, n)
    rel_close(run_matmul(la, ctx, kernels, f"matmul_nt_{fmt}_into", a, raw, m, k, n), want, 1e-3, f"{fmt} m={m} k={k} n={n}")
    if fmt == "q4_0":
        rel_close(run_matmul(la, ctx, kernels, "matmul_nt_q4_0_f32out_into", a, raw, m, k, n, f32out=True), want, 5e-4, "f32 out")
    device_status_ok(kernels)


@pytest.mark.parametrize("hd,n_q,n_kv,bits,total,window,ring", [
    (128, 8, 1, 2, 33, 0, 0), (128, 8, 1, 3, 1025, 0, 0), (128, 12, 2, 4, 2600, 0, 0), (512, 8, 1, 2, 17, 0, 0),
    (512, 6, 2, 3, 700, 300, 0), (512, 4, 2, 4, 513, 0, 0), (256, 5, 1, 3, 1600, 512, 512), (256, 10, 1, 4, 4097, 0, 0)])
def test_code_attention_head_sizes_and_code_widths(la, orc, ctx, kernels, hd, n_q, n_kv, bits, total, window, ring):
    c = Cache(la, orc, ctx, hd, n_kv, bits, ring or total, seed=41 + total)
    c.fill_single(total, ring)
    kc, kn, vc, vn, lv, _ = c.device()
    rq = orc.hadamard_rotate(la.synth.normal(43, n_q * hd).astype(np.float32), c.signs, hd, n_q, True, False)
    out = Guarded(la, ctx, n_q * hd * 4)
    b = la.CommandBatch.new(ctx)
    kernels.flash_attention_tq_into(b, la.CudaBuffer.from_slice(ctx, rq), kc, kn, vc, vn, lv, out.view, hd, total, total - 1,
                                    n_q, n_kv, window, bits, ring, 0.0625)
    b.commit_and_wait()
    want = orc.flash_attention_tq(rq, c.kc, c.kn, c.vc, c.vn, c.levels, hd, total, total - 1, n_q, n_kv, window, bits, ring, 0.0625)
    rel_close(out.read(np.float32), want, 1e-3, "attention over codes")


@pytest.mark.parametrize("hd,n_q,n_kv,bits", [(256, 8, 1, 4), (128, 8, 2, 2)])
def test_ragged_pool_attention_in_work_items(la, orc, ctx, kernels, hd, n_q, n_kv, bits):
    """Pools of ten lanes or more and over 2048 keys: lanes are cut into items that the CTAs draw.  Twice with the same
    object: the draw's counters are back at zero."""
    cap = 2600
    positions = np.array([0, 31, 255, 256, 700, 1023, 2047, 2048, 2598, 2599, 5, 1800], np.uint32)
    n = positions.size
    c = Cache(la, orc, ctx, hd, n_kv, bits, n * cap, seed=90)
    c.fill_pool(positions, cap, 0)
    kc, kn, vc, vn, lv, sg = c.device()
    q = la.synth.normal_f16((n, n_q, hd), 91)
    want = orc.tq_attention_fused(q, c.kc, c.kn, c.vc, c.vn, c.levels, c.signs, positions, hd, cap, n_q, n_kv, 0, bits, n, 0, 0.0625)
    outs = []
    for _ in range(2):
        out = Guarded(la, ctx, n * n_q * hd * 2)
        b = la.CommandBatch.new(ctx)
        kernels.tq_attention_batched_into(b, la.CudaBuffer.from_slice(ctx, q), kc, kn, vc, vn, lv, sg, out.view,
                                          la.CudaBuffer.from_slice(ctx, positions), hd, cap, n_q, n_kv, 0, bits, n, 0, 0.0625)
        b.commit_and_wait()
        outs.append(out.read(np.float16))
        rel_close(outs[-1], want.astype(np.float32), 2e-3, "ragged pool")
    assert np.array_equal(outs[0].view(np.uint16), outs[1].view(np.uint16))


@pytest.mark.parametrize("hd,bits,cap", [(64, 3, 700), (512, 2, 1100)])
def test_merge_of_many_rows(la, orc, ctx, kernels, hd, bits, cap):
    """A warp per row: over 296 (lane, head) rows whose partials a second launch adds up, at the head sizes that the other
    tests do not bring there (an output that 16-byte stores cannot reach keeps the first launch from merging)."""
    n, n_q, n_kv = 41, 8, 1
    positions = (np.arange(n, dtype=np.uint32) * 7) % 90
    positions[[3, 17, 40]] = cap - 1
    c = Cache(la, orc, ctx, hd, n_kv, bits, n * cap, seed=95)
    c.fill_pool(positions, cap, 0)
    kc, kn, vc, vn, lv, sg = c.device()
    q = la.synth.normal_f16((n, n_q, hd), 96)
    want = orc.tq_attention_fused(q, c.kc, c.kn, c.vc, c.vn, c.levels, c.signs, positions, hd, cap, n_q, n_kv, 0, bits, n, 0, 0.0625)
    nbytes = n * n_q * hd * 2
    buf = la.CudaBuffer.empty(ctx, nbytes + 8)
    b = la.CommandBatch.new(ctx)
    kernels.tq_attention_batched_into(b, la.CudaBuffer.from_slice(ctx, q), kc, kn, vc, vn, lv, sg,
                                      la.CudaBuffer.wrap(ctx, buf.device_ptr + 8, nbytes), la.CudaBuffer.from_slice(ctx, positions), hd, cap,
                                      n_q, n_kv, 0, bits, n, 0, 0.0625)
    assert b.dispatch_count() == 2
    b.commit_and_wait()
    rel_close(buf.as_slice(np.uint8)[8:].view(np.float16), want.astype(np.float32), 2e-3, "merge of many rows")


# 128 rows (query rows x heads, heads rounded up to a power of two) to a tile, 32 or 64 keys to a step; chunks of enough rows
# that the prefill kernel is the one that runs, and one that is too small for it
@pytest.mark.parametrize("hd,n_q,n_kv,bits,rows,start,window", [
    (256, 8, 1, 2, 150, 463, 0), (256, 8, 1, 4, 300, 500, 128), (256, 3, 1, 3, 300, 31, 0), (256, 16, 2, 2, 155, 1000, 512),
    (128, 8, 2, 3, 160, 95, 0), (128, 12, 1, 4, 161, 300, 64), (128, 2, 1, 2, 310, 1, 0), (256, 8, 1, 4, 33, 500, 128)])
def test_prefill_attention_at_tile_edges(la, orc, ctx, kernels, hd, n_q, n_kv, bits, rows, start, window):
    total = start + rows
    c = Cache(la, orc, ctx, hd, n_kv, bits, total, seed=60 + total)
    c.fill_single(total, 0)
    kc, kn, vc, vn, lv, sg = c.device()
    q = la.synth.normal_f16((rows, n_q, hd), 61)
    rq = orc.hadamard_rotate(q.astype(np.float32), c.signs, hd, rows * n_q, True, False)
    want = orc.flash_attention_tq_prefill(rq, c.kc, c.kn, c.vc, c.vn, c.levels, hd, total, start, rows, n_q, n_kv, window, bits, 0, 0.0625)
    out, fused = Guarded(la, ctx, rows * n_q * hd * 4), Guarded(la, ctx, rows * n_q * hd * 2)
    b = la.CommandBatch.new(ctx)
    kernels.flash_attention_tq_prefill_into(b, la.CudaBuffer.from_slice(ctx, rq), kc, kn, vc, vn, lv, out.view, hd, total, start, rows,
                                            n_q, n_kv, window, bits, 0, 0.0625)
    kernels.tq_attention_prefill_into(b, la.CudaBuffer.from_slice(ctx, q), kc, kn, vc, vn, lv, sg, fused.view, hd, total, start, rows,
                                      n_q, n_kv, window, bits, 0, 0.0625)
    b.commit_and_wait()
    rel_close(out.read(np.float32), want, 1e-3, "prefill")
    back = orc.hadamard_rotate(want, c.signs, hd, rows * n_q, False, True)
    rel_close(fused.read(np.float16), back.astype(np.float16).astype(np.float32), 2e-3, "fused prefill")
    device_status_ok(kernels)


@pytest.mark.parametrize("hd,n_q,n_kv,total,window", [(64, 8, 1, 1, 0), (64, 6, 2, 1001, 0), (128, 16, 1, 63, 0), (256, 8, 1, 8191, 0),
                                                      (512, 8, 2, 129, 0), (256, 7, 1, 700, 333)])
def test_f16_attention_at_odd_lengths(la, orc, ctx, kernels, hd, n_q, n_kv, total, window):
    q, k, v = f16_case(la, hd, n_q, n_kv, total, 71)
    out = Guarded(la, ctx, n_q * hd * 2)
    f = lambda x: la.CudaBuffer.from_slice(ctx, x)
    if window:
        kernels.attention_sliding(ctx, f(q), f(k), f(v), out.view, hd, total, total - 1, window, n_q, n_kv)
    else:
        b = la.CommandBatch.new(ctx)
        kernels.flash_decoding_into(ctx, b, f(q), f(k), f(v), out.view, hd, total, total - 1, n_q, n_kv)
        b.commit_and_wait()
    rel_close(out.read(np.float16), orc.attention_f16(q, k, v, hd, total, total - 1, n_q, n_kv, window).astype(np.float32), 2e-3, "f16")


# the caller's partial buffers: at any float, refused at less
@pytest.mark.parametrize("offset", [0, 4, 8, 12, 2])
def test_windowed_split_with_partials_at_any_float(la, orc, ctx, kernels, offset):
    hd, n_q, n_kv, total, window = 256, 8, 1, 700, 333
    q, k, v = f16_case(la, hd, n_q, n_kv, total, 72)
    splits = kernels.flash_split_count(window)
    bufs = [la.CudaBuffer.empty(ctx, 16 + n_q * splits * d * 4) for d in (1, 1, hd)]
    parts = [la.CudaBuffer.wrap(ctx, b.device_ptr + offset, b.nbytes - 16) for b in bufs]
    out = Guarded(la, ctx, n_q * hd * 2)
    f = lambda x: la.CudaBuffer.from_slice(ctx, x)
    b = la.CommandBatch.new(ctx)
    call = lambda: kernels.flash_attention_windowed_split_into(b, f(q), f(k), f(v), out.view, *parts, hd, total, total - 1, n_q, n_kv, window, splits)
    if offset % 4:
        with pytest.raises(la.Error) as ei:
            call()
        assert ei.value.kind == "InvalidArgument"
        b.commit_and_wait()
        return
    call()
    b.commit_and_wait()
    rel_close(out.read(np.float16), orc.attention_f16(q, k, v, hd, total, total - 1, n_q, n_kv, window).astype(np.float32), 2e-3, "windowed split")


@pytest.mark.parametrize("hd", [128, 256, 512])
@pytest.mark.parametrize("rows", [1, 7, 9, 65])
def test_encoder_rows_at_block_edges(la, orc, ctx, kernels, hd, rows):
    bits, n_kv = 2 + rows % 3, 1
    levels, signs = la.tq_levels(hd, bits), la.tq_signs(hd, la.TQ_SEED)
    x = la.synth.normal_f16((rows, n_kv, hd), 81)
    cb = la.tq_code_bytes(hd, bits)
    want_c, want_n = np.zeros(rows * cb, np.uint8), np.zeros(rows, np.float16)
    orc.encode_kv(x, levels, signs, want_c, want_n, hd, n_kv, rows, bits, 0, 0)
    codes, norms = gpu_encode(la, ctx, kernels, x, levels, signs, hd, n_kv, rows, bits, 0, 0, rows)
    assert np.array_equal(codes, want_c) and np.array_equal(norms, want_n.view(np.uint16))


# V rows far above unit norm and logits that grow along the context: P, the softmax weight times v_norm * gamma, is stored as
# f16, so the weights that a lagging maximum allows (up to e^8) must not carry it past 65504
@pytest.mark.parametrize("bits,vnorm,window,ring", [(2, 1000.0, 0, 0), (2, 60000.0, 512, 1024), (4, 1000.0, 0, 0), (4, 200.0, 512, 1024),
                                                    (3, 60000.0, 0, 0)])
def test_prefill_attention_keeps_large_value_norms_in_range(la, orc, ctx, kernels, bits, vnorm, window, ring):
    hd, n_q, n_kv, rows, total = 256, 8, 1, 400, 1200
    slots = ring or total
    levels, signs = la.tq_levels(hd, bits), la.tq_signs(hd, la.TQ_SEED)
    cb = la.tq_code_bytes(hd, bits)
    rng = np.random.default_rng(bits)
    one = rng.integers(0, 256, cb, dtype=np.uint8)                      # every K row has one direction; its norms set the logits
    k0 = levels[(np.unpackbits(one, bitorder="little").reshape(hd, bits) * (1 << np.arange(bits))).sum(1)].astype(np.float64)
    slot = np.arange(total) % slots                                     # (later positions overwrite the ring's earlier ones)
    kc, vc = np.tile(one, slots), rng.integers(0, 256, slots * cb, dtype=np.uint8)
    kn, vn = np.zeros(slots, np.float16), np.zeros(slots, np.float16)
    kn[slot] = (0.5 + np.arange(total) / total + 6.0 * (np.arange(total) % 240 >= 130)).astype(np.float16)   # steps of 4.5 .. 6.9
    vn[slot] = np.where(np.arange(total) // 100 % 2, vnorm, 1.0).astype(np.float16)
    rq = (np.linspace(0.75, 1.15, rows * n_q)[:, None] * (k0 / (k0 @ k0))).astype(np.float32).reshape(-1)   # logits 0.4 .. 8.6
    q16 = orc.hadamard_rotate(rq, signs, hd, rows * n_q, False, True).astype(np.float16)
    f = lambda a: la.CudaBuffer.from_slice(ctx, a)
    bufs = (f(kc), f(kn), f(vc), f(vn), f(levels))
    out, fused = Guarded(la, ctx, rows * n_q * hd * 4), Guarded(la, ctx, rows * n_q * hd * 2)
    start = total - rows
    b = la.CommandBatch.new(ctx)
    kernels.flash_attention_tq_prefill_into(b, f(rq), *bufs, out.view, hd, total, start, rows, n_q, n_kv, window, bits, ring, 1.0)
    kernels.tq_attention_prefill_into(b, f(q16), *bufs, f(signs), fused.view, hd, total, start, rows, n_q, n_kv, window, bits, ring, 1.0)
    b.commit_and_wait()
    attend = lambda x: orc.flash_attention_tq_prefill(x, kc, kn, vc, vn, levels, hd, total, start, rows, n_q, n_kv, window, bits, ring, 1.0)
    # The weights sum to 1.  tq2 rounds each P to f16: 2^-11 of it.  tq3 / tq4 keep P, levels and query in two f16 parts, 2^-22 each;
    # of logits up to 8.6 that is 2^-19, and 2^-16 leaves as much again for f32 sums and exponentials.  The inverse rotation keeps
    # a row's 2-norm, and its f16 result adds 2^-11.
    most = np.abs(levels).max() * vnorm
    tol = most * (2.0 ** -11 if bits == 2 else 2.0 ** -16)
    got, want = out.read(np.float32), attend(rq)
    assert np.isfinite(got).all() and np.abs(got - want).max() <= tol, np.abs(got - want).max() / tol
    back = orc.hadamard_rotate(attend(orc.hadamard_rotate(q16.astype(np.float32), signs, hd, rows * n_q, True, False)), signs, hd, rows * n_q, False, True)
    back, got = back.reshape(-1, hd), fused.read(np.float16).astype(np.float64).reshape(-1, hd)
    off = np.linalg.norm(got - back, axis=1)
    assert np.all(off <= tol * np.sqrt(hd) + 2.0 ** -11 * np.linalg.norm(back, axis=1)), off.max()
    device_status_ok(kernels)


# The same for the decode kernel, where the maximum may lag if P has two parts (all but tq2 at head_dim 256): one split per lane stored as it is,
# splits merged in a cluster, splits and a merge launch, and work items.  A warp takes every eighth tile, so logits that step every 256 keys
# (128 at head_dim 512) step along its tiles: by less than the lag, so that weights stay well above 1, past it, and down again.
DECODE_FORMS = [   # head_dim, bits, form, lanes (0: a single one), rows of a lane, largest V norm
    (128, 2, "one", 100, 1800, 1.0), (128, 3, "items", 80, 4200, 60000.0), (128, 4, "cluster", 60, 2000, 85.0), (128, 4, "merge", 60, 2000, 1000.0),
    (256, 2, "items", 80, 4200, 60000.0), (256, 3, "cluster", 60, 2000, 60000.0), (256, 4, "items", 80, 4200, 121.0), (256, 4, "one", 100, 1800, 1000.0),
    (256, 4, "merge", 0, 100000, 200.0), (512, 2, "merge", 60, 2000, 60000.0), (512, 3, "items", 50, 4200, 200.0), (512, 4, "cluster", 60, 2000, 60000.0)]


@pytest.mark.parametrize("hd,bits,form,lanes,cap,vnorm", DECODE_FORMS)
def test_decode_attention_keeps_large_value_norms_in_range(la, orc, ctx, kernels, hd, bits, form, lanes, cap, vnorm):
    n_q, n = 8, max(lanes, 1)
    levels, signs = la.tq_levels(hd, bits), la.tq_signs(hd, la.TQ_SEED)
    cb = la.tq_code_bytes(hd, bits)
    rng = np.random.default_rng(bits)
    decode = lambda codes: levels[(np.unpackbits(codes.reshape(-1, cb), axis=1, bitorder="little").reshape(-1, hd, bits) * (1 << np.arange(bits))).sum(2)].astype(np.float64)
    one = rng.integers(0, 256, cb, dtype=np.uint8)                      # every K row has one direction; its norms set the logits
    k0 = decode(one)[0]
    at = np.arange(cap)
    step = np.array([0.5, 5.2, 0.8, 7.9, 1.4, 8.3, 6.0, 0.6])[at // (128 if hd == 512 else 256) % 8] + 6.0 * (at // 2048 % 2)
    kn = np.tile((step + at % 7 / 20).astype(np.float16), n)
    vn = np.tile(np.array([1.0, vnorm, 1.0, vnorm / 8, 1.0], np.float32)[at // 64 % 5].astype(np.float16), n)
    kc, vc = np.tile(one, n * cap), rng.integers(0, 256, n * cap * cb, dtype=np.uint8)
    positions = np.full(n, cap - 1, np.uint32)
    if n > 1:
        positions[1::2] = rng.integers(0, cap, positions[1::2].size)
    rq = (np.linspace(0.75, 1.15, n * n_q)[rng.permutation(n * n_q)][:, None] * (k0 / (k0 @ k0))).astype(np.float32)   # logits 0.4 .. 16.9
    q16 = orc.hadamard_rotate(rq.reshape(-1), signs, hd, n * n_q, False, True).astype(np.float16)
    f = lambda a: la.CudaBuffer.from_slice(ctx, a)
    bufs, pos, rows = (f(kc), f(kn), f(vc), f(vn), f(levels)), f(positions), n * n_q
    shift = 8 if form == "merge" else 0   # (an output that 16-byte stores cannot reach keeps the first launch from merging)
    outs = [la.CudaBuffer.from_slice(ctx, np.full(shift + rows * hd * e + 256, 0xA5, np.uint8)) for e in (4, 2)]
    views = [la.CudaBuffer.wrap(ctx, o.device_ptr + shift, rows * hd * e) for o, e in zip(outs, (4, 2))]
    launches = []
    for fused in (False, True):
        b = la.CommandBatch.new(ctx)
        if lanes and fused:
            kernels.tq_attention_batched_into(b, f(q16), *bufs, f(signs), views[1], pos, hd, cap, n_q, 1, 0, bits, n, 0, 1.0)
        elif lanes:
            kernels.flash_attention_tq_batched_into(b, f(rq), *bufs, views[0], pos, hd, cap, n_q, 1, 0, bits, n, 0, 1.0)
        elif fused:
            kernels.tq_attention_into(b, f(q16), *bufs, f(signs), views[1], hd, cap, cap - 1, n_q, 1, 0, bits, 0, 1.0)
        else:
            kernels.flash_attention_tq_into(b, f(rq), *bufs, views[0], hd, cap, cap - 1, n_q, 1, 0, bits, 0, 1.0)
        launches.append(b.dispatch_count())
        b.commit_and_wait()
    assert launches == ([1, 1] if form in ("one", "cluster") else [2, 2])   # (of an aligned output, two are items and their merge)

    def attend(x):   # in 64 bits
        out = np.empty((n, n_q, hd))
        for i, p in enumerate(positions):
            rows_i = slice(i * cap, i * cap + int(p) + 1)
            s = (x.astype(np.float64).reshape(n, n_q, hd)[i] @ k0)[:, None] * kn[rows_i].astype(np.float64)
            w = np.exp(s - s.max(1, keepdims=True))
            w /= w.sum(1, keepdims=True)
            out[i] = (w * vn[rows_i].astype(np.float64)) @ decode(vc.reshape(-1, cb)[rows_i].copy())
        return out.reshape(-1, hd)

    # The weights sum to 1, and their errors count twice, in the sum and in its divisor.  tq2 at head_dim 256 rounds each P to f16: 2^-11 of it,
    # and holds levels to 2^-18.  The others keep P, levels and query in two f16 parts, 2^-22 each, and a logit is a chain of head_dim / 16
    # MMAs of up to 2^-23 of what is summed so far, half of the result in the mean: (head_dim / 16 + 4) 2^-24 of logits up to 17.  64 2^-24
    # leaves room for f32 sums over a warp's tiles and for exponentials.  The inverse rotation keeps a row's 2-norm; its f16 result adds 2^-11.
    most = np.abs(levels).max() * max(vnorm, 1.0)
    tol = 2.0 * most * ((17.0 * (hd / 16 + 4) + 64.0) * 2.0 ** -24 + (2.0 ** -11 if bits == 2 and hd == 256 else 0.0))
    raw = [o.as_slice(np.uint8) for o in outs]
    assert all((r[:shift] == 0xA5).all() and (r[r.size - 256:] == 0xA5).all() for r in raw)
    got, want = raw[0][shift:-256].view(np.float32).reshape(-1, hd), attend(rq)
    assert np.isfinite(got).all() and np.abs(got - want).max() <= tol, np.abs(got - want).max() / tol
    rotated = orc.hadamard_rotate(q16.astype(np.float32).reshape(-1), signs, hd, rows, True, False)
    back = orc.hadamard_rotate(attend(rotated).astype(np.float32).reshape(-1), signs, hd, rows, False, True).reshape(-1, hd)
    got = raw[1][shift:-256].view(np.float16).astype(np.float64).reshape(-1, hd)
    off = np.linalg.norm(got - back, axis=1)
    assert np.all(off <= tol * np.sqrt(hd) + 2.0 ** -11 * np.linalg.norm(back, axis=1)), off.max()
    device_status_ok(kernels)


# Q4_0 at 17 .. 64 rows goes to the kernel that is estimated to take less: shapes of both, their clusters and edges
Q4_0_ROUTES = [(17, 1024, 8200), (24, 4096, 4600), (32, 1536, 4100), (20, 256, 19001), (29, 768, 20737), (33, 128, 75777), (64, 256, 75900),
               (45, 384, 19300), (32, 2048, 12300), (18, 160, 334)]


@pytest.mark.parametrize("m,k,n", Q4_0_ROUTES)
def test_q4_0_matmul_of_17_to_64_rows(la, orc, ctx, kernels, m, k, n):
    raw = la.synth.q4_0_weights(n, k, 33)
    a = la.synth.normal_f16((m, k), 34)
    got = run_matmul(la, ctx, kernels, "matmul_nt_q4_0_into", a, raw, m, k, n).reshape(m, n)
    rows = np.r_[0:200, n // 2:n // 2 + 200, n - 200:n] if n > 4000 else np.arange(n)   # (the oracle's time)
    some = np.ascontiguousarray(raw.reshape(n, -1)[rows])
    want = orc.matmul_nt(orc.Q4_0, a, some, m, k, rows.size).reshape(m, -1)
    rel_close(got[:, rows], want, 1e-3, f"q4_0 m={m} k={k} n={n}")
    assert np.isfinite(got).all() and got.std(axis=0).min() > 0
    device_status_ok(kernels)


@pytest.mark.parametrize("m,k,n", [(17, 6144, 1536), (40, 1536, 6144), (64, 800, 3000)])
def test_q4_0_matmul_with_f32_output_keeps_its_precision(la, orc, ctx, kernels, m, k, n):
    """f32 outputs at 17 .. 64 rows: sums of f32-scaled 32-k blocks, K / 32 roundings of 2^-24 each in a walk, sqrt(192) 2^-24 = 8e-7 at
    the most and 1e-7 as a rule; the tcgen05 accumulators are 9e-7 off."""
    raw, a = la.synth.q4_0_weights(n, k, 35), la.synth.normal_f16((m, k), 36)
    got = run_matmul(la, ctx, kernels, "matmul_nt_q4_0_f32out_into", a, raw, m, k, n, f32out=True).astype(np.float64)
    want = orc.matmul_nt(orc.Q4_0, a, raw, m, k, n).astype(np.float64).reshape(m, n)
    assert np.linalg.norm(got - want) <= 3e-7 * np.linalg.norm(want), np.linalg.norm(got - want) / np.linalg.norm(want)


@pytest.mark.parametrize("m,k,n", [(24, 512, 40000), (20, 256, 100000), (50, 256, 150000), (24, 4096, 6144), (40, 1536, 6144)])
def test_q4_0_matmul_of_17_to_64_rows_is_not_the_slower_kernel(la, ctx, kernels, monkeypatch, m, k, n):
    """The choice against the register-direct kernel alone (LOCAL_CUDA_DECODE_TC=0): at most 1.1 times its time, where a wrong
    choice takes 1.16 to 1.9 times."""
    monkeypatch.setenv("LOCAL_CUDA_DECODE_TC", "0")
    other = la.Kernels.new(ctx)
    w, x, out = la.CudaBuffer.empty(ctx, n * k // 32 * 18), la.CudaBuffer.empty(ctx, m * k * 2), la.CudaBuffer.empty(ctx, m * n * 2)
    w.zero(), x.zero()
    graphs = []
    for kern in (kernels, other):
        for begin in (la.CommandBatch.new, la.CommandBatch.capture):
            b = begin(ctx)
            for _ in range(20):
                kern.matmul_nt_q4_0_into(b, x, w, out, m, k, n)
            b.commit_and_wait() if begin == la.CommandBatch.new else graphs.append(b.end_capture())
    best = [np.inf, np.inf]
    for _ in range(8):
        for i, g in enumerate(graphs):
            ctx.synchronize()
            t = time.perf_counter()
            g.launch()
            ctx.synchronize()
            best[i] = min(best[i], time.perf_counter() - t)
    for g in graphs:
        g.destroy()
    other.close()
    assert best[0] <= 1.1 * best[1], best


@pytest.mark.parametrize("m,k,n", [(24, 512, 32000), (24, 896, 44000), (64, 192, 44000), (20, 768, 64000), (24, 384, 40000), (48, 256, 150000)])
def test_q4_0_matmul_of_17_to_64_rows_is_the_faster_of_two_kernels(la, ctx, kernels, monkeypatch, m, k, n):
    """The choice against either kernel alone (LOCAL_CUDA_DECODE_TC=0: register-direct, LOCAL_CUDA_DECODE_MMA=0: large-batch): at most 1.1 times the faster
    one's time, at shapes where the other takes up to 1.33 times that."""
    kerns = [kernels]
    for off in ("LOCAL_CUDA_DECODE_TC", "LOCAL_CUDA_DECODE_MMA"):
        monkeypatch.setenv(off, "0")
        kerns.append(la.Kernels.new(ctx))
        monkeypatch.delenv(off)
    w, x, out = la.CudaBuffer.empty(ctx, n * k // 32 * 18), la.CudaBuffer.empty(ctx, m * k * 2), la.CudaBuffer.empty(ctx, m * n * 2)
    w.zero(), x.zero()
    graphs, best = [], [np.inf] * 3
    for kern in kerns:
        for begin in (la.CommandBatch.new, la.CommandBatch.capture):
            b = begin(ctx)
            for _ in range(20):
                kern.matmul_nt_q4_0_into(b, x, w, out, m, k, n)
            b.commit_and_wait() if begin == la.CommandBatch.new else graphs.append(b.end_capture())
    for _ in range(8):
        for i, g in enumerate(graphs):
            ctx.synchronize()
            t = time.perf_counter()
            g.launch()
            ctx.synchronize()
            best[i] = min(best[i], time.perf_counter() - t)
    for g in graphs:
        g.destroy()
    for kern in kerns[1:]:
        kern.close()
    assert best[0] <= 1.1 * min(best[1:]), best


# Chunks that only the estimate of the kernels' times sends to the prefill kernel, and single lanes that it cuts into more splits than one launch merges
@pytest.mark.parametrize("hd,n_q,n_kv,bits,rows,start,window", [
    (128, 8, 1, 2, 64, 4000, 0), (256, 8, 1, 3, 24, 8100, 0), (256, 8, 1, 4, 100, 1900, 0), (128, 4, 1, 4, 40, 5000, 0), (128, 8, 2, 4, 130, 700, 300),
    (256, 8, 1, 2, 1, 4200, 0), (128, 16, 1, 3, 1, 6677, 0), (512, 8, 1, 4, 1, 4100, 0)])
def test_attention_of_two_launches(la, orc, ctx, kernels, hd, n_q, n_kv, bits, rows, start, window):
    total = start + rows
    c = Cache(la, orc, ctx, hd, n_kv, bits, total, seed=70 + total)
    c.fill_single(total, 0)
    kc, kn, vc, vn, lv, sg = c.device()
    q = la.synth.normal_f16((rows, n_q, hd), 62)
    rq = orc.hadamard_rotate(q.astype(np.float32), c.signs, hd, rows * n_q, True, False)
    want = orc.flash_attention_tq_prefill(rq, c.kc, c.kn, c.vc, c.vn, c.levels, hd, total, start, rows, n_q, n_kv, window, bits, 0, 0.0625)
    out, fused = Guarded(la, ctx, rows * n_q * hd * 4), Guarded(la, ctx, rows * n_q * hd * 2)
    f = lambda x: la.CudaBuffer.from_slice(ctx, x)
    b = la.CommandBatch.new(ctx)
    if rows > 1:
        kernels.flash_attention_tq_prefill_into(b, f(rq), kc, kn, vc, vn, lv, out.view, hd, total, start, rows, n_q, n_kv, window, bits, 0, 0.0625)
        kernels.tq_attention_prefill_into(b, f(q), kc, kn, vc, vn, lv, sg, fused.view, hd, total, start, rows, n_q, n_kv, window, bits, 0, 0.0625)
    else:
        kernels.flash_attention_tq_into(b, f(rq), kc, kn, vc, vn, lv, out.view, hd, total, start, n_q, n_kv, window, bits, 0, 0.0625)
        kernels.tq_attention_into(b, f(q), kc, kn, vc, vn, lv, sg, fused.view, hd, total, start, n_q, n_kv, window, bits, 0, 0.0625)
    assert b.dispatch_count() == 4
    b.commit_and_wait()
    rel_close(out.read(np.float32), want, 1e-3, "two launches")
    back = orc.hadamard_rotate(want, c.signs, hd, rows * n_q, False, True)
    rel_close(fused.read(np.float16), back.astype(np.float16).astype(np.float32), 2e-3, "two launches, fused")
    device_status_ok(kernels)


@pytest.mark.parametrize("hd,bits,less,more", [(128, 2, (64, 8192), (128, 8192)), (256, 4, (128, 2000), (256, 2000)), (128, 4, (128, 2000), (256, 2000)),
                                               (256, 3, (64, 4096), (128, 4096)), (128, 3, (1, 7000), (1, 16000)), (256, 4, (1, 6000), (1, 16000))])
def test_attention_over_less_takes_no_longer(la, ctx, kernels, hd, bits, less, more):
    """Fewer rows over the same keys, and fewer keys: at most 1.1 times as long, where a form chosen by a wrong estimate took up to 1.6 times."""
    cb, (rows, total) = la.tq_code_bytes(hd, bits), more
    zeros = lambda n: la.CudaBuffer.empty(ctx, n)
    kc, kn, vc, vn = zeros(total * cb), zeros(total * 2), zeros(total * cb), zeros(total * 2)
    lv, sg = la.CudaBuffer.from_slice(ctx, la.tq_levels(hd, bits)), la.CudaBuffer.from_slice(ctx, la.tq_signs(hd, la.TQ_SEED))
    q, out = zeros(rows * 8 * hd * 2), zeros(rows * 8 * hd * 2)
    graphs, best = [], [np.inf] * 2
    for n, keys in (less, more):
        def call(b):
            if n > 1:
                kernels.tq_attention_prefill_into(b, q, kc, kn, vc, vn, lv, sg, out, hd, keys, keys - n, n, 8, 1, 0, bits, 0, 0.0625)
            else:
                kernels.tq_attention_into(b, q, kc, kn, vc, vn, lv, sg, out, hd, keys, keys - 1, 8, 1, 0, bits, 0, 0.0625)
        for begin in (la.CommandBatch.new, la.CommandBatch.capture):
            b = begin(ctx)
            for _ in range(20):
                call(b)
            b.commit_and_wait() if begin == la.CommandBatch.new else graphs.append(b.end_capture())
    for _ in range(8):
        for i, g in enumerate(graphs):
            ctx.synchronize()
            t = time.perf_counter()
            g.launch()
            ctx.synchronize()
            best[i] = min(best[i], time.perf_counter() - t)
    for g in graphs:
        g.destroy()
    assert best[0] <= 1.1 * best[1], best


@pytest.mark.parametrize("bits,rows,start", [(2, 256, 768), (4, 150, 1900)])
def test_prefill_attention_captured_without_an_eager_call_first(la, orc, ctx, bits, rows, start):
    """The prefill kernel's partials need scratch memory, which cannot grow while a graph is recorded: with none reserved the
    chunk takes the decode kernel, which merges its splits itself.  After an eager call the graph holds the prefill kernel."""
    hd, n_q, n_kv = 256, 8, 1
    c = Cache(la, orc, ctx, hd, n_kv, bits, start + rows, seed=77)
    c.fill_single(start + rows, 0)
    kc, kn, vc, vn, lv, sg = c.device()
    q = la.CudaBuffer.from_slice(ctx, la.synth.normal_f16((rows, n_q, hd), 78))
    rq = orc.hadamard_rotate(q.as_slice(np.float16).astype(np.float32), c.signs, hd, rows * n_q, True, False)
    want = orc.flash_attention_tq_prefill(rq, c.kc, c.kn, c.vc, c.vn, c.levels, hd, start + rows, start, rows, n_q, n_kv, 0, bits, 0, 0.0625)
    back = orc.hadamard_rotate(want, c.signs, hd, rows * n_q, False, True).astype(np.float16).astype(np.float32)
    k = la.Kernels.new(ctx)
    launches = []
    for eager_first in (False, True):
        out = Guarded(la, ctx, rows * n_q * hd * 2)
        call = lambda b: k.tq_attention_prefill_into(b, q, kc, kn, vc, vn, lv, sg, out.view, hd, start + rows, start, rows, n_q, n_kv, 0, bits, 0, 0.0625)
        if eager_first:
            b = la.CommandBatch.new(ctx)
            call(b)
            b.commit_and_wait()
        b = la.CommandBatch.capture(ctx)
        call(b)
        launches.append(b.dispatch_count())
        graph = b.end_capture()
        graph.launch()
        ctx.synchronize()
        rel_close(out.read(np.float16), back, 2e-3, "captured prefill")
        graph.destroy()
    assert launches == [1, 2]
    k.close()


def test_expired_wait_in_prefill_attention_reports_timeout(la, orc, ctx, monkeypatch):
    """LOCAL_CUDA_TEST_WAIT_EXPIRY=1: the prefill kernel's "keys ready" barrier expects an arrival nobody makes and its waits have a
    short limit.  The launch returns, the status word reads Timeout, and a regular kernels object works afterwards."""
    import ctypes as C
    hd, n_q, n_kv, bits, rows, start = 256, 8, 1, 2, 150, 463
    c = Cache(la, orc, ctx, hd, n_kv, bits, start + rows, seed=75)
    c.fill_single(start + rows, 0)
    kc, kn, vc, vn, lv, sg = c.device()
    q = la.synth.normal_f16((rows, n_q, hd), 76)
    monkeypatch.setenv("LOCAL_CUDA_TEST_WAIT_EXPIRY", "1")
    expiring = la.Kernels.new(ctx)
    monkeypatch.delenv("LOCAL_CUDA_TEST_WAIT_EXPIRY")
    regular = la.Kernels.new(ctx)
    out = Guarded(la, ctx, rows * n_q * hd * 2)
    for k in (expiring, regular):
        b = la.CommandBatch.new(ctx)
        k.tq_attention_prefill_into(b, la.CudaBuffer.from_slice(ctx, q), kc, kn, vc, vn, lv, sg, out.view, hd, start + rows, start, rows, n_q,
                                    n_kv, 0, bits, 0, 0.0625)
        b.commit_and_wait()   # returns: no wait is endless
        if k is expiring:
            st = C.c_int(0)
            with pytest.raises(la.Error) as ei:
                k.kernels_device_status(C.addressof(st))
            assert ei.value.kind == "Timeout" and st.value != 0
    rq = orc.hadamard_rotate(q.astype(np.float32), c.signs, hd, rows * n_q, True, False)
    want = orc.flash_attention_tq_prefill(rq, c.kc, c.kn, c.vc, c.vn, c.levels, hd, start + rows, start, rows, n_q, n_kv, 0, bits, 0, 0.0625)
    back = orc.hadamard_rotate(want, c.signs, hd, rows * n_q, False, True)
    rel_close(out.read(np.float16), back.astype(np.float16).astype(np.float32), 2e-3, "after an expired wait")
    device_status_ok(regular)
    expiring.close()
    regular.close()


# Branches of the prefill kernel beside the usual one: signs other than +-1 (its query transform by shuffles), and rings, in which
# a key tile wraps
@pytest.mark.parametrize("hd,n_q,n_kv,bits,rows,start,window,ring,unit", [
    (256, 8, 1, 2, 150, 463, 0, 0, False), (128, 8, 2, 3, 160, 95, 0, 0, False), (256, 8, 1, 4, 300, 500, 128, 0, False),
    (128, 8, 1, 2, 310, 40, 0, 0, False),
    (256, 8, 1, 2, 400, 1500, 512, 1024, True), (256, 8, 1, 4, 300, 777, 128, 512, True), (128, 12, 1, 3, 330, 1001, 200, 560, True),
    (256, 8, 1, 2, 400, 1500, 512, 1024, False)])
def test_prefill_attention_with_other_signs_and_rings(la, orc, ctx, kernels, hd, n_q, n_kv, bits, rows, start, window, ring, unit):
    total = start + rows
    c = Cache(la, orc, ctx, hd, n_kv, bits, ring or total, seed=70 + total)
    c.fill_single(total, ring)
    kc, kn, vc, vn, lv, _ = c.device()
    signs = c.signs if unit else (c.signs * np.linspace(0.5, 1.5, hd)).astype(np.float32)
    q = la.synth.normal_f16((rows, n_q, hd), 71)
    rq = orc.hadamard_rotate(q.astype(np.float32), signs, hd, rows * n_q, True, False)
    want = orc.flash_attention_tq_prefill(rq, c.kc, c.kn, c.vc, c.vn, c.levels, hd, total, start, rows, n_q, n_kv, window, bits, ring, 0.0625)
    out, fused = Guarded(la, ctx, rows * n_q * hd * 4), Guarded(la, ctx, rows * n_q * hd * 2)
    b = la.CommandBatch.new(ctx)
    kernels.flash_attention_tq_prefill_into(b, la.CudaBuffer.from_slice(ctx, rq), kc, kn, vc, vn, lv, out.view, hd, total, start, rows,
                                            n_q, n_kv, window, bits, ring, 0.0625)
    kernels.tq_attention_prefill_into(b, la.CudaBuffer.from_slice(ctx, q), kc, kn, vc, vn, lv, la.CudaBuffer.from_slice(ctx, signs), fused.view,
                                      hd, total, start, rows, n_q, n_kv, window, bits, ring, 0.0625)
    b.commit_and_wait()
    rel_close(out.read(np.float32), want, 1e-3, "prefill")
    back = orc.hadamard_rotate(want, signs, hd, rows * n_q, False, True)
    rel_close(fused.read(np.float16), back.astype(np.float16).astype(np.float32), 2e-3, "fused prefill")
    device_status_ok(kernels)


@pytest.mark.parametrize("hd,rows,total", [(128, 0, 700), (512, 0, 700), (128, 0, 5000), (128, 256, 900)])
def test_two_bit_attention_keeps_its_weights_in_32_bits(la, orc, ctx, kernels, hd, rows, total):
    """At head_dim 128 and 512 tq2 attention ran with f32 levels and weights on CUDA cores; on tensor cores they are an f16 and the f16
    of the remainder, 2^-22 of each.  An average over N keys of both signs is sqrt(N) times smaller than its terms, so 5000 keys turn
    that into 2^-22 * 71 = 1.7e-5 at the very most (were all of it one way), and f32 sums stay below it: 1e-5 of the result's norm,
    where weights in one f16 leave 2e-4."""
    n_q, n_kv, bits = 8, 1, 2
    c = Cache(la, orc, ctx, hd, n_kv, bits, total, seed=79)
    c.fill_single(total, 0)
    kc, kn, vc, vn, lv, _ = c.device()
    rq = orc.hadamard_rotate(la.synth.normal(80, max(rows, 1) * n_q * hd).astype(np.float32), c.signs, hd, max(rows, 1) * n_q, True, False)
    out = la.CudaBuffer.empty(ctx, rq.size * 4)
    b = la.CommandBatch.new(ctx)
    head = (b, la.CudaBuffer.from_slice(ctx, rq), kc, kn, vc, vn, lv, out, hd, total)
    if rows:
        kernels.flash_attention_tq_prefill_into(*head, total - rows, rows, n_q, n_kv, 0, bits, 0, 0.0625)
        want = orc.flash_attention_tq_prefill(rq, c.kc, c.kn, c.vc, c.vn, c.levels, hd, total, total - rows, rows, n_q, n_kv, 0, bits, 0, 0.0625)
    else:
        kernels.flash_attention_tq_into(*head, total - 1, n_q, n_kv, 0, bits, 0, 0.0625)
        want = orc.flash_attention_tq(rq, c.kc, c.kn, c.vc, c.vn, c.levels, hd, total, total - 1, n_q, n_kv, 0, bits, 0, 0.0625)
    b.commit_and_wait()
    off = out.as_slice(np.float32).astype(np.float64) - want
    assert np.linalg.norm(off) <= 1e-5 * np.linalg.norm(want.astype(np.float64)), np.linalg.norm(off) / np.linalg.norm(want)
