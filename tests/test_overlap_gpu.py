"""Launches of one batch that run beside each other where their buffers do not meet (LcOrder in csrc/lc_internal.h): any sequence of
projections gives, bit for bit, what the same calls give with a wait after each."""
import numpy as np
import pytest

from test_matvec_gpu import device_status_ok

pytestmark = pytest.mark.gpu
K = 1024


def calls(rng, n_inputs, n_views, n_weights, count):
    """(input, weight, output) triples; inputs 0 .. n_inputs - 1 are never written, the rest are the output views."""
    out = []
    for _ in range(count):
        o = int(rng.integers(n_views))
        i = int(rng.integers(n_inputs)) if rng.random() < 0.6 else n_inputs + int(rng.integers(n_views))
        out.append((i, int(rng.integers(n_weights)), o))
    return out


@pytest.mark.parametrize("m,fmt", [(1, "q4_0"), (1, "tq2_0"), (7, "tq2_0"), (16, "q4_0"), (16, "tq2_0"), (33, "tq2_0"), (64, "tq2_0"), (24, "q4_0"), (64, "q4_0"),
                                   (100, "tq2_0"), (100, "q4_0")])
@pytest.mark.parametrize("captured", [False, True])
def test_same_as_one_after_the_other(la, ctx, kernels, m, fmt, captured):
    """Random chains over a few inputs, weights and output views.  Views overlap each other by half and are inputs of later calls, so
    reads after writes, writes after reads and writes after writes all occur, next to runs without any."""
    rng = np.random.default_rng(100 * m + len(fmt) + captured)
    make = la.synth.q4_0_weights if fmt == "q4_0" else la.synth.tq2_0_weights
    op = getattr(kernels, ("matvec_%s_into" if m == 1 else "matmul_nt_%s_into") % fmt)
    weights = [la.CudaBuffer.from_slice(ctx, make(K, K, seed=50 + i)) for i in range(5)]
    inputs = [la.CudaBuffer.from_slice(ctx, (la.synth.normal_f16((m, K), 60 + i) * np.float16(0.25)).astype(np.float16)) for i in range(3)]
    bytes_ = m * K * 2
    half = (bytes_ // 2) & ~15
    slab = la.CudaBuffer.empty(ctx, 10 * bytes_)
    # 0 .. 3 apart from each other, 4 and 5 lie across two of them
    views = [la.CudaBuffer.wrap(ctx, slab.device_ptr + at, bytes_) for at in (0, bytes_, 2 * bytes_, 3 * bytes_, half, 2 * bytes_ + half)]
    seq = calls(rng, len(inputs), len(views), len(weights), 60)
    seq += [(i % 3, i % 5, i % 4) for i in range(12)]                      # a run without a conflict until it comes round
    seq += [(0, i % 5, 0) if i % 2 else (len(inputs), i % 5, 1) for i in range(8)]   # each reads what the one before wrote

    def one(b, c):
        i, w, o = c
        x, out = (inputs + views)[i], views[o]
        if i - len(inputs) == o or (i >= len(inputs) and {i - len(inputs), o} in ({4, 0}, {4, 1}, {5, 2}, {5, 3})):
            x = inputs[0]                                                  # (a call's own operands do not overlap)
        if m == 1:
            op(b, weights[w], x, out, K, K)
        else:
            op(b, x, weights[w], out, m, K, K)

    slab.zero()
    for c in seq:
        b = la.CommandBatch.new(ctx)
        one(b, c)
        b.commit_and_wait()
    want = slab.as_slice(np.uint16).copy()
    for _ in range(4):
        slab.zero()
        if captured:
            b = la.CommandBatch.capture(ctx)
            for c in seq:
                one(b, c)
            graph = b.end_capture()
            graph.launch()
            ctx.synchronize()
            graph.destroy()
        else:
            b = la.CommandBatch.new(ctx)
            for c in seq:
                one(b, c)
            b.commit_and_wait()
        assert np.array_equal(slab.as_slice(np.uint16), want)
    assert np.any(want)
    device_status_ok(kernels)


def test_other_launches_end_a_run(la, ctx, kernels):
    """Between projections on disjoint buffers stand launches that declare nothing (additions, one in place): what follows them sees
    their results, and they see those of every projection before."""
    m, n = 16, 8192
    x = la.CudaBuffer.from_slice(ctx, la.synth.normal_f16((m, K), 70))
    ws = [la.CudaBuffer.from_slice(ctx, la.synth.tq2_0_weights(n, K, seed=80 + i)) for i in range(4)]
    outs = [la.CudaBuffer.empty(ctx, m * n * 2) for _ in range(4)]
    total, copy = la.CudaBuffer.empty(ctx, m * n * 2), la.CudaBuffer.empty(ctx, m * n * 2)

    def run(wait):
        for o in outs + [total, copy]:
            o.zero()
        b = la.CommandBatch.new(ctx)
        step = lambda: (b.commit_and_wait(), la.CommandBatch.new(ctx))[1] if wait else b
        for r in range(3):
            for i in range(4):
                kernels.matmul_nt_tq2_0_into(b, x, ws[(i + r) % 4], outs[i], m, K, n)
                b = step()
            kernels.residual_add_into(b, outs[r], outs[3], total, m * n)
            b = step()
            kernels.matmul_nt_tq2_0_into(b, x, ws[r], outs[3], m, K, n)    # overwrites what the addition read
            b = step()
            kernels.residual_add_into(b, total, copy, copy, m * n)
            b = step()
        b.commit_and_wait()
        return [o.as_slice(np.uint16).copy() for o in outs + [total, copy]]

    want = run(True)
    for _ in range(5):
        for a, b in zip(run(False), want):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("work", ["none", "copy", "upload", "download", "zero", "fill", "as_slice", "from_bytes", "alloc", "gather", "graph", "add"])
def test_order_behind_other_work(la, ctx, kernels, work):
    """A matmul runs beside those before it only while nothing but matmuls stands between: behind every other kind of work on the stream it
    waits, also where that work declares no buffers of its own."""
    m, n = 16, 4096
    x = la.CudaBuffer.from_slice(ctx, la.synth.normal_f16((m, K), 95))
    ws = [la.CudaBuffer.from_slice(ctx, la.synth.tq2_0_weights(n, K, seed=96 + i)) for i in range(3)]
    outs = [la.CudaBuffer.empty(ctx, m * n * 2) for _ in range(4)]
    other = la.CudaBuffer.empty(ctx, m * n * 2)
    host = np.zeros(m * n, np.uint16)
    if work == "gather":
        import torch  # noqa: F401  (brings the NCCL that it links; the system's, loaded first, would be in its way)
    comm = la.Communicator(ctx, la.Communicator.unique_id(), 0, 1) if work == "gather" else None
    b = la.CommandBatch.capture(ctx)
    kernels.residual_add_into(b, other, other, other, m * n)
    graph = b.end_capture()
    b = la.CommandBatch.new(ctx)
    kernels.residual_add_into(b, other, other, other, m * n)
    orders = []
    for i in range(3):
        kernels.matmul_nt_tq2_0_into(b, x, ws[i], outs[i], m, K, n)
        orders.append(b.last_order())
    assert orders == [0, 1, 2]
    {"none": lambda: None,
     "copy": lambda: b.blit_buffer_copy(outs[2], 0, other, 0, m * n * 2),
     "upload": lambda: b.upload(other, 0, host.ctypes.data, m * n * 2),
     "download": lambda: b.download(outs[2], 0, host.ctypes.data, m * n * 2),
     "zero": lambda: other.zero(),
     "fill": lambda: other.fill(1),
     "as_slice": lambda: outs[2].as_slice(np.uint16),
     "from_bytes": lambda: other.copy_from_bytes(host),
     "alloc": lambda: la.CudaBuffer.empty(ctx, 4096),
     "gather": lambda: comm.all_gather_into(b, outs[2], 0, other, m * n * 2),
     "graph": lambda: graph.launch(),
     "add": lambda: kernels.residual_add_into(b, other, other, other, m * n)}[work]()
    kernels.matmul_nt_tq2_0_into(b, x, ws[0], outs[3], m, K, n)
    assert b.last_order() == (2 if work == "none" else 0)
    b.commit_and_wait()
    graph.destroy()
    if comm:
        comm.close()


def test_no_runs_once_the_stream_is_out(la):
    own = la.CudaContext.new(0)
    kernels = la.Kernels.new(own)
    x, w = la.CudaBuffer.from_slice(own, la.synth.normal_f16((16, K), 97)), la.CudaBuffer.from_slice(own, la.synth.tq2_0_weights(4096, K, seed=98))
    outs = [la.CudaBuffer.empty(own, 16 * 4096 * 2) for _ in range(3)]

    def orders():
        b, got = la.CommandBatch.new(own), []
        for o in outs:
            kernels.matmul_nt_tq2_0_into(b, x, w, o, 16, K, 4096)
            got.append(b.last_order())
        b.commit_and_wait()
        return got

    assert orders()[1:] == [1, 2]
    assert own.stream
    assert orders() == [0, 0, 0]
    own.set_overlap(True)
    assert orders() == [0, 1, 2]
    for o in outs + [x, w]:
        o.free()
    kernels.close()
    own.close()


def test_weights_written_two_dispatches_before(la, ctx, kernels):
    """Constant operands written by a dispatch with another in between, where both are projections that run beside others: the launch behind the run
    starts when all of them are complete."""
    m, n = 16, 4096
    x = la.CudaBuffer.from_slice(ctx, la.synth.normal_f16((m, K), 90))
    ws = [la.CudaBuffer.from_slice(ctx, la.synth.tq2_0_weights(n, K, seed=91 + i)) for i in range(6)]
    outs = [la.CudaBuffer.empty(ctx, m * n * 2) for _ in range(6)]
    normed = la.CudaBuffer.empty(ctx, m * K * 2)
    norm_w = la.CudaBuffer.wrap(ctx, outs[4].device_ptr, K * 2)          # the norm's weights: what the projection before last wrote

    def run(wait):
        for o in outs + [normed]:
            o.zero()
        b = la.CommandBatch.new(ctx)
        for i in range(6):
            kernels.matmul_nt_tq2_0_into(b, x, ws[i], outs[i], m, K, n)
            if wait:
                b.commit_and_wait()
                b = la.CommandBatch.new(ctx)
        kernels.rms_norm_into(b, x, norm_w, normed, K, m, 1e-6)
        b.commit_and_wait()
        return normed.as_slice(np.uint16).copy()

    want = run(True)
    assert np.any(want)
    for _ in range(10):
        assert np.array_equal(run(False), want)
