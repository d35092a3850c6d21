"""The decode step in 64 bits without a rounding between its operations (numpy): what the kernels' forms of it are compared with where
the question is how much their own arithmetic adds.  Sequence: local-engine/src/layer.rs:731-868."""
import numpy as np


def _fwht(x):
    """Orthonormal Walsh-Hadamard transform of the last axis."""
    d, shape = x.shape[-1], x.shape
    x, n = x.reshape(-1, d), 1
    while n < d:
        x = x.reshape(-1, d // (2 * n), 2, n)
        x = np.stack((x[:, :, 0] + x[:, :, 1], x[:, :, 0] - x[:, :, 1]), axis=2).reshape(-1, d)
        n *= 2
    return (x / np.sqrt(d)).reshape(shape)


def _rms(x, w, eps):
    return x / np.sqrt((x * x).mean(-1, keepdims=True) + eps) * w


def _rope(x, pos, theta):
    half = x.shape[-1] // 2
    ang = pos * theta ** (-np.arange(half) / half)
    a, b, c, s = x[..., :half], x[..., half:], np.cos(ang), np.sin(ang)
    return np.concatenate((a * c - b * s, b * c + a * s), -1)


class Step64:
    def __init__(self, orc, cfg, layers, emb, final_norm, geometry):
        self.cfg, self.geo = cfg, geometry
        hd, qd, kd = cfg.head_dim, cfg.n_q_heads * cfg.head_dim, cfg.n_kv_heads * cfg.head_dim
        shapes = {"wq": (qd, cfg.hidden), "wk": (kd, cfg.hidden), "wv": (kd, cfg.hidden), "wo": (cfg.hidden, qd),
                  "wgate": (cfg.inter, cfg.hidden), "wup": (cfg.inter, cfg.hidden), "wdown": (cfg.hidden, cfg.inter)}
        self.layers = [{n: orc.expand_f32(orc.TQ2_0, t, *shapes[n]).reshape(shapes[n]).astype(np.float64) if n in shapes else t.astype(np.float64)
                        for n, t in layer.items()} for layer in layers]
        self.emb = orc.expand_f32(orc.Q4_0, emb, cfg.vocab, cfg.hidden).reshape(cfg.vocab, cfg.hidden).astype(np.float64)
        self.final_norm = final_norm.astype(np.float64)
        self.levels, self.signs = orc.tq_levels(hd, cfg.kv_bits).astype(np.float64), orc.tq_signs(hd, 0x7459C0DE).astype(np.float64)

    def rows(self, codes, norms):
        """Rotated rows from packed codes [n, code bytes] and norms [n]."""
        bits = self.cfg.kv_bits
        u = np.unpackbits(codes, axis=1, bitorder="little").reshape(len(codes), self.cfg.head_dim, bits) @ (1 << np.arange(bits))
        return self.levels[u] * norms.astype(np.float64)[:, None]

    def encoded(self, x):
        """Rotated rows of x [n, head_dim] as the cache keeps them: nearest levels, the norm in f16."""
        norm = np.sqrt((x * x).sum(-1, keepdims=True))
        r = _fwht(x / norm * self.signs)
        return self.levels[np.abs(r[..., None] - self.levels).argmin(-1)] * norm.astype(np.float16).astype(np.float64)

    def step(self, pools, tokens, positions):
        """Logits of every lane; pools (as OracleModel.pools) are read only."""
        c = self.cfg
        hd, nq, nkv = c.head_dim, c.n_q_heads, c.n_kv_heads
        out = []
        for lane, (token, pos) in enumerate(zip(tokens, positions)):
            pos = int(pos)
            x = self.emb[int(token)] * c.embed_scale
            for L, pool, (rows, ring, window) in zip(self.layers, pools, self.geo):
                h = _rms(x, L["attn_norm"], c.rms_eps)
                q = _rope(_rms((L["wq"] @ h).reshape(nq, hd), L["q_norm"], c.rms_eps), pos, c.rope_theta)
                k = _rope(_rms((L["wk"] @ h).reshape(nkv, hd), L["k_norm"], c.rms_eps), pos, c.rope_theta)
                v = _rms((L["wv"] @ h).reshape(nkv, hd), 1.0, c.rms_eps)
                rq, nk, nv = _fwht(q * self.signs) * c.softmax_scale, self.encoded(k), self.encoded(v)
                begin = max(0, pos + 1 - window) if window else 0
                keys = np.arange(begin, pos)
                at = (lane * rows + (keys % ring if ring else keys))[:, None] * nkv + np.arange(nkv)
                o = np.empty((nq, hd))
                for g in range(nkv):
                    kr, vr = ((self.rows(pool[n + "_codes"].reshape(-1, hd * c.kv_bits // 8)[at[:, g]], pool[n + "_norms"][at[:, g]])) for n in "kv")
                    kr, vr = np.vstack((kr, nk[g])), np.vstack((vr, nv[g]))
                    mine = slice(g * nq // nkv, (g + 1) * nq // nkv)
                    s = rq[mine] @ kr.T
                    p = np.exp(s - s.max(-1, keepdims=True))
                    o[mine] = _fwht(p / p.sum(-1, keepdims=True) @ vr) * self.signs
                x = x + _rms(L["wo"] @ o.reshape(-1), L["post_attn_norm"], c.rms_eps)
                h = _rms(x, L["ffn_norm"], c.rms_eps)
                gate, up = L["wgate"] @ h, L["wup"] @ h
                inner = np.clip(np.sqrt(2 / np.pi) * (gate + 0.044715 * gate ** 3), -10, 10)
                x = x + _rms(L["wdown"] @ (0.5 * gate * (1 + np.tanh(inner)) * up), L["post_ffn_norm"], c.rms_eps)
            out.append(self.emb @ _rms(x, self.final_norm, c.rms_eps))
        return np.array(out)
