"""The merge of many splits of few heads by a cluster per head (csrc/split_merge.cuh), at its edges: the fewest splits it takes, counts that
eight does not divide, more splits than keys, every head_dim and the most heads; against the CPU oracle at the attention tests' tolerances
(1e-3 for f32 outputs, 2e-3 for f16 ones)."""
import numpy as np
import pytest

from gpu_util import Guarded, rel_close
from test_attention_gpu import Cache, f16_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd,n_q,n_kv,total,splits,skew", [(256, 8, 2, 3000, 31, 0), (256, 8, 2, 3000, 32, 0), (256, 8, 1, 3001, 33, 1), (64, 4, 1, 2500, 257, 0),
                                                           (128, 18, 2, 2000, 64, 0), (512, 2, 2, 1500, 100, 1), (512, 8, 1, 200, 300, 0), (256, 1, 1, 40, 1000, 0)])
def test_f16_rows(la, orc, ctx, kernels, hd, n_q, n_kv, total, splits, skew):
    q, k, v = f16_case(la, hd, n_q, n_kv, total, 600 + splits)
    out = Guarded(la, ctx, n_q * hd * 2)
    pm, ps = la.CudaBuffer.empty(ctx, n_q * splits * 4), la.CudaBuffer.empty(ctx, n_q * splits * 4)
    raw = la.CudaBuffer.empty(ctx, (n_q * splits * hd + 1) * 4)
    pa = la.CudaBuffer.wrap(ctx, raw.device_ptr + 4 * skew, n_q * splits * hd * 4)
    b = la.CommandBatch.new(ctx)
    kernels.flash_attention_windowed_split_into(b, la.CudaBuffer.from_slice(ctx, q), la.CudaBuffer.from_slice(ctx, k), la.CudaBuffer.from_slice(ctx, v),
                                                out.view, pm, ps, pa, hd, total, total - 1, n_q, n_kv, 0, splits)
    assert b.dispatch_count() == 2
    b.commit_and_wait()
    rel_close(out.read(np.float16), orc.attention_f16(q, k, v, hd, total, total - 1, n_q, n_kv, 0).astype(np.float32), 2e-3, "f16 rows")


@pytest.mark.parametrize("hd,n_q,n_kv,bits,total", [(256, 8, 1, 2, 32768), (256, 8, 1, 4, 9001), (128, 8, 1, 3, 9000), (512, 8, 1, 2, 7001), (64, 18, 2, 4, 9999)])
def test_codes(la, orc, ctx, kernels, hd, n_q, n_kv, bits, total):
    c = Cache(la, orc, ctx, hd, n_kv, bits, total, seed=total)
    c.fill_single(total, 0)
    kc, kn, vc, vn, lv, sg = c.device()
    q16 = la.synth.normal_f16((n_q, hd), 59)
    rq = orc.hadamard_rotate(q16.astype(np.float32).ravel(), c.signs, hd, n_q, True, False)
    plain, fused = Guarded(la, ctx, n_q * hd * 4), Guarded(la, ctx, n_q * hd * 2)
    b = la.CommandBatch.new(ctx)
    kernels.flash_attention_tq_into(b, la.CudaBuffer.from_slice(ctx, rq), kc, kn, vc, vn, lv, plain.view, hd, total, total - 1, n_q, n_kv, 0, bits, 0, 0.0625)
    kernels.tq_attention_into(b, la.CudaBuffer.from_slice(ctx, q16), kc, kn, vc, vn, lv, sg, fused.view, hd, total, total - 1, n_q, n_kv, 0, bits, 0, 0.0625)
    b.commit_and_wait()
    want = orc.flash_attention_tq(rq, c.kc, c.kn, c.vc, c.vn, c.levels, hd, total, total - 1, n_q, n_kv, 0, bits, 0, 0.0625)
    rel_close(plain.read(np.float32), want, 1e-3, "rotated")
    want = orc.tq_attention_fused(q16, c.kc, c.kn, c.vc, c.vn, c.levels, c.signs, None, hd, 0, n_q, n_kv, 0, bits, 1, 0, 0.0625, total, total - 1)
    rel_close(fused.read(np.float16), want.astype(np.float32), 2e-3, "fused")
