"""The routed-expert decoder (f32 host-path conventions, GGUF Q8_0 attention + Q4_K expert banks): the
oracle's token step against an independent float64 restatement on CPU, and (GPU) the device decoder
against the oracle through the C ABI."""
import numpy as np
import pytest

from oracle import oracle as O
from stark_b200 import synthetic as S


def _dense(kind, blocks, rows, columns):
    """GGUF rows decoded through the pinned block decoder, as float64."""
    blocks = np.ascontiguousarray(blocks, np.uint8).reshape(rows, -1)
    return np.stack([O.gguf_decode_row(kind, blocks[r], columns) for r in range(rows)]).astype(np.float64)


class _Float64Decoder:
    """The same token step in float64 numpy with dense weights: no shared code with the C restatement beyond
    the block decoder.  Sums are numpy's, not sequential, so agreement is to rounding, not to the bit."""

    def __init__(self, cfg, w):
        self.c = cfg
        H, D, E, I = cfg["hidden"], cfg["head_dim"], cfg["experts"], cfg["inter"]
        qd, kd = cfg["q_heads"] * D, cfg["kv_heads"] * D
        self.table = _dense(8, w["token_table"], cfg["vocab"], H)
        self.output = _dense(8, w["output"], cfg["vocab"], H)
        self.final = w["final_norm"].astype(np.float64)
        self.layers = []
        for l in w["layers"]:
            self.layers.append(dict(
                qkv=_dense(8, l["qkv"], qd + 2 * kd, H), o=_dense(8, l["o"], H, qd), router=l["router"].astype(np.float64),
                gate=_dense(12, l["gate"], E * I, H).reshape(E, I, H), up=_dense(12, l["up"], E * I, H).reshape(E, I, H),
                down=_dense(12, l["down"], E * H, I).reshape(E, H, I),
                **{k: l[k].astype(np.float64) for k in ("attn_norm", "ffn_norm", "q_norm", "k_norm")}))
        self.keys = [[] for _ in w["layers"]]
        self.values = [[] for _ in w["layers"]]
        self.experts = []

    def _norm(self, x, w):
        return x / np.sqrt(np.mean(x * x) + self.c["eps"]) * w

    def _rope(self, head, position):
        d = head.size
        i = np.arange(d // 2)
        angle = position * self.c["rope_theta"] ** (-(2.0 * i) / d)
        a, b = head[:d // 2].copy(), head[d // 2:].copy()
        return np.concatenate([a * np.cos(angle) - b * np.sin(angle), a * np.sin(angle) + b * np.cos(angle)])

    def step(self, token):
        c = self.c
        D, QH, KV = c["head_dim"], c["q_heads"], c["kv_heads"]
        position = len(self.keys[0])
        x = self.table[token].copy()
        self.experts = []
        for li, l in enumerate(self.layers):
            n = self._norm(x, l["attn_norm"])
            qkv = l["qkv"] @ n
            q, k, v = qkv[:QH * D].reshape(QH, D), qkv[QH * D:(QH + KV) * D].reshape(KV, D), qkv[(QH + KV) * D:].reshape(KV, D)
            q = np.stack([self._rope(self._norm(h, l["q_norm"]), position) for h in q])
            k = np.stack([self._rope(self._norm(h, l["k_norm"]), position) for h in k])
            self.keys[li].append(k)
            self.values[li].append(v)
            K, V = np.stack(self.keys[li]), np.stack(self.values[li])  # [t, kv, d]
            att = np.empty((QH, D))
            for h in range(QH):
                g = h // (QH // KV)
                s = K[:, g] @ q[h] / np.sqrt(D)
                p = np.exp(s - s.max())
                att[h] = (p / p.sum()) @ V[:, g]
            x = x + l["o"] @ att.reshape(-1)
            n = self._norm(x, l["ffn_norm"])
            scores = l["router"] @ n
            ids = sorted(range(c["experts"]), key=lambda e: (-scores[e], e))[:c["active"]]
            p = np.exp(scores[ids] - scores[ids].max())
            p /= p.sum()
            mix = np.zeros_like(x)
            for e, pe in zip(ids, p):
                g = l["gate"][e] @ n
                mix += pe * (l["down"][e] @ (g / (1.0 + np.exp(-g)) * (l["up"][e] @ n)))
            x = x + mix
            self.experts.append(ids)
        return self.output @ self._norm(x, self.final)


def test_oracle_step_matches_float64_restatement():
    cfg = S.MOE_CONFIGS["moe-tiny"]
    w = S.moe_weights(cfg, seed=3)
    oracle, exact = O.MoEDecoder(cfg, w, 16, threads=2), _Float64Decoder(cfg, w)
    for token in (5, 400, 5, 77, 123):
        got, want = oracle.step(token), exact.step(token)
        assert oracle.last_experts.tolist() == exact.experts
        assert np.abs(got - want).max() <= 2e-5 * max(1.0, np.abs(want).max())
    assert oracle.position == 5
    with pytest.raises(ValueError):
        oracle.step(cfg["vocab"])


def test_rope_matches_the_closed_form():
    """ripple.rs:653-666: pairs (i, i + d/2) rotate by position * theta^(-2i/d)."""
    head = np.arange(1, 9, dtype=np.float32)
    out = head.copy()
    f = O.lib().so_rope_f32
    import ctypes as C
    f.restype, f.argtypes = None, [C.c_void_p, C.c_uint32, C.c_uint32, C.c_float]
    f(out.ctypes.data, 8, 3, 10000.0)
    for i in range(4):
        ang = 3.0 * 10000.0 ** (-(2.0 * i) / 8.0)
        assert abs(out[i] - (head[i] * np.cos(ang) - head[i + 4] * np.sin(ang))) < 1e-5
        assert abs(out[i + 4] - (head[i] * np.sin(ang) + head[i + 4] * np.cos(ang))) < 1e-5
    same = head.copy()
    f(same.ctypes.data, 8, 0, 10000.0)
    assert same.tolist() == head.tolist()                                    # position 0 is the identity


def _close(got, want, bound=2e-4):
    return np.abs(got - want).max() <= bound * max(1.0, np.abs(want).max())


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["moe-tiny", "moe-small", "moe-a3b-layers"])
def test_device_decoder_matches_oracle(name):
    from stark_b200.engine import MoEModel
    cfg = S.MOE_CONFIGS[name]
    w = S.moe_weights(cfg, seed=1)
    context = 192
    model, oracle = MoEModel.load(cfg, w, context), O.MoEDecoder(cfg, w, context)
    prompt = S.prompt(cfg, 40, seed=2)
    # token by token: logits, routing and the greedy pick
    agree = 0
    for t in prompt[:12]:
        got, want = model.step(int(t)), oracle.step(int(t))
        assert np.isfinite(got).all() and _close(got, want)
        assert model.last_experts().tolist() == oracle.last_experts.tolist()
        agree += int(got.argmax() == want.argmax())
    assert agree >= 11
    # cache-only prompt rows, then a step: same as stepping through them
    model.ingest(prompt[12:])
    oracle.ingest(prompt[12:])
    assert model.position == oracle.position == 40
    got, want = model.step(9), oracle.step(9)
    assert _close(got, want)
    # greedy decode chained on the device follows the oracle's own greedy decode while no near-tie parts them
    first = int(want.argmax())
    picks = model.generate_greedy(first, 16)
    token, same = first, 0
    for i in range(16):
        lg = oracle.step(token)
        token = int(lg.argmax())
        same += int(picks[i] == token)
        if picks[i] != token:
            break
    assert same >= 8, (same, picks)
    assert model.position == 57
    # teacher-forced: both decoders are fed the oracle's greedy tokens, top-1 must agree on >= 99 % of 100 steps
    model.reset()
    oracle.reset()
    model.ingest(prompt[:-1])
    oracle.ingest(prompt[:-1])
    token, agree, steps = int(prompt[-1]), 0, 100
    for i in range(steps):
        got, want = model.step(token), oracle.step(token)
        assert _close(got, want, 1e-3)   # absolute tolerance on the f32 logits: 1e-3 of the largest magnitude
        agree += int(got.argmax() == want.argmax())
        token = int(want.argmax())
    assert agree >= 99, agree
    assert model.position == 39 + steps
    # reset: the first step reproduces itself bit for bit
    model.reset()
    a = model.step(int(prompt[0]))
    model.reset()
    b = model.step(int(prompt[0]))
    assert model.position == 1 and a.tobytes() == b.tobytes()
    assert model.launches_per_token >= 4 + 8 * cfg["layers"]
    model.close()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["moe-small", "moe-a3b-layers"])
def test_fused_hand_offs_change_no_bit(name, monkeypatch):
    """The residual add + norm inside the router kernel and the per-head norm + rope inside the attention kernel
    form their sums in the order of the separate kernels: logits, experts and tokens are the same bits."""
    from stark_b200.engine import MoEModel
    cfg = S.MOE_CONFIGS[name]
    w = S.moe_weights(cfg, seed=4)
    prompt = S.prompt(cfg, 70, seed=6)
    seen = []
    for fuse in ("1", "0"):
        monkeypatch.setenv("STARK_B200_MOE_FUSE", fuse)
        model = MoEModel.load(cfg, w, 128)
        assert model.launches_per_token == 4 + (8 if fuse == "1" else 10) * cfg["layers"]
        model.ingest(prompt[:-1])
        logits = model.step(int(prompt[-1]))
        experts = model.last_experts().tolist()
        picks = model.generate_greedy(int(logits.argmax()), 12)
        seen.append((logits.tobytes(), experts, picks.tolist(), model.step(3).tobytes()))
        model.close()
    assert seen[0] == seen[1]


@pytest.mark.gpu
@pytest.mark.parametrize("name,portions", [
    ("moe-tiny", (2,)), ("moe-tiny", (1, 3, 2)), ("moe-tiny", (511, 1, 5)), ("moe-tiny", (515,)), ("moe-small", (15, 16, 17)),
    ("moe-small", (31, 2)), ("moe-a3b-layers", (4, 33)), ("moe-a3b-layers", (129,))])
def test_prompt_rows_in_passes(name, portions):
    """Portions around a tile's rows and a pass's, behind rows already in the cache: the step that follows and the experts of
    the last ingested row are the oracle's."""
    from stark_b200.engine import MoEModel
    cfg = S.MOE_CONFIGS[name]
    w = S.moe_weights(cfg, seed=5)
    context = sum(portions) + 4
    model, oracle = MoEModel.load(cfg, w, context), O.MoEDecoder(cfg, w, context)
    ids = S.prompt(cfg, sum(portions) + 2, seed=9)
    at = 0
    for n in portions:
        model.ingest(ids[at:at + n])
        oracle.ingest(ids[at:at + n])
        at += n
        assert model.position == at
        assert model.last_experts().tolist() == oracle.last_experts.tolist()
    for t in ids[at:]:
        got, want = model.step(int(t)), oracle.step(int(t))
        assert _close(got, want)
        assert model.last_experts().tolist() == oracle.last_experts.tolist()
    model.close()


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,portions", [
    (dict(), (2, 15, 16, 17, 3, 515)),                                                                     # passes of every raggedness
    (dict(hidden=2048, q_heads=32, kv_heads=4, experts=128, active=8, inter=768), (33, 260)),             # spans of 16 rows and more
    (dict(hidden=4352, inter=4864, experts=5, active=3, q_heads=34, kv_heads=17), (18,)),                 # rows of more slices than warps
    (dict(hidden=8192, inter=256, experts=300, active=32, q_heads=8, kv_heads=1), (5, 40)),               # the widest; most picks
    (dict(hidden=768, inter=512, experts=129, active=1, q_heads=10, kv_heads=5), (17, 1020))])
def test_rows_of_a_pass_leave_a_tokens_bits(sizes, portions):
    """A prompt in portions, and its rows one by one (as ranks of a group take them): the same logits, experts and tokens."""
    from stark_b200.engine import MoEModel
    cfg = dict(S.MOE_CONFIGS["moe-tiny"], **sizes)
    w = S.moe_weights(cfg, seed=21)
    context = sum(portions) + 8
    ids = S.prompt(cfg, context, seed=31)
    seen = []
    for single in (False, True):
        model, at, out = MoEModel.load(cfg, w, context), 0, []
        for n in portions:
            for part in ([ids[i:i + 1] for i in range(at, at + n)] if single else [ids[at:at + n]]):
                model.ingest(part)
            at += n
            out.append(model.last_experts().tobytes())
        out += [model.step(int(ids[at])).tobytes(), model.last_experts().tobytes(), model.generate_greedy(int(ids[at + 1]), 4).tobytes()]
        seen.append(out)
        model.close()
    assert seen[0] == seen[1]


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [
    dict(hidden=8192), dict(hidden=8448), dict(hidden=12288), dict(hidden=12544), dict(q_heads=96, kv_heads=12), dict(q_heads=98, kv_heads=49),
    dict(inter=12288), dict(inter=12544)])
def test_prompt_rows_of_the_widest_models(sizes):
    """Row widths at the most that a pass of rows takes and one step past it: rows go one by one then, and input rows of q, k, v
    and o past the matvec's own bound are refused.  12 288 columns are the 48 KB of shared memory a launch has unasked."""
    from stark_b200._lib import StarkB200Error
    from stark_b200.engine import MoEModel
    cfg = dict(S.MOE_CONFIGS["moe-tiny"], layers=2, experts=4, active=2, **sizes)
    w = S.moe_weights(cfg, seed=12)
    model, oracle = MoEModel.load(cfg, w, 24), O.MoEDecoder(cfg, w, 24)
    ids = S.prompt(cfg, 19, seed=2)
    if max(cfg["hidden"], 128 * cfg["q_heads"]) > 12288:
        for call in (lambda: model.ingest(ids[:1]), lambda: model.ingest(ids[:-1])):
            with pytest.raises(StarkB200Error, match="unsupported"):
                call()
        model.close()
        return
    model.ingest(ids[:-1])
    oracle.ingest(ids[:-1])
    assert model.position == 18
    assert model.last_experts().tolist() == oracle.last_experts.tolist()
    assert _close(model.step(int(ids[-1])), oracle.step(int(ids[-1])))
    model.close()


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,behind", [
    (dict(hidden=4608, inter=4352, experts=4, active=3, q_heads=2, kv_heads=1), 0),    # rows of more super-blocks than warps
    (dict(hidden=256, inter=256, experts=300, active=32, q_heads=8, kv_heads=2), 15),  # one warp a row tile; most picks
    (dict(hidden=768, inter=512, experts=129, active=1, q_heads=10, kv_heads=5), 17),  # ragged teams; one score past 128
    (dict(hidden=256, inter=256, experts=8, active=2, q_heads=8, kv_heads=1), 1023),   # spans grow from 16 rows to 17
])
def test_token_kernels_at_their_edges(sizes, behind):
    """Tokens behind rows of the cache against the oracle, and a second model of the same weights to the bit."""
    from stark_b200.engine import MoEModel
    cfg = dict(S.MOE_CONFIGS["moe-tiny"], **sizes)
    w = S.moe_weights(cfg, seed=8)
    models = [MoEModel.load(cfg, w, behind + 3) for _ in range(2)]
    oracle = O.MoEDecoder(cfg, w, behind + 3)
    ids = S.prompt(cfg, behind + 3, seed=3)
    for m in models:
        m.ingest(ids[:behind])
    oracle.ingest(ids[:behind])
    for t in ids[behind:]:
        got, again, want = models[0].step(int(t)), models[1].step(int(t)), oracle.step(int(t))
        assert got.tobytes() == again.tobytes()
        assert _close(got, want)
        assert models[0].last_experts().tolist() == oracle.last_experts.tolist()
    for m in models:
        m.close()


@pytest.mark.gpu
def test_device_decoder_refuses_bad_calls():
    from stark_b200._lib import StarkB200Error
    from stark_b200.engine import MoEModel
    cfg = S.MOE_CONFIGS["moe-tiny"]
    w = S.moe_weights(cfg, seed=4)
    model = MoEModel(cfg, 4)
    with pytest.raises(StarkB200Error):                                      # nothing loaded yet
        model.step(1)
    model.set_globals(w["token_table"], w["output"], w["final_norm"])
    for i, l in enumerate(w["layers"]):
        model.set_layer(i, l)
    with pytest.raises(StarkB200Error):
        model.step(cfg["vocab"])
    with pytest.raises(StarkB200Error):
        model.ingest([1, 2, 3, 4, 5])                                        # more rows than the cache holds
    model.ingest([1, 2, 3])
    model.step(4)
    with pytest.raises(StarkB200Error):
        model.step(5)                                                        # the cache is full
    assert model.position == 4
    bad = dict(w["layers"][0])
    bad["attn_norm"] = np.full(cfg["hidden"], np.nan, np.float32)
    with pytest.raises(StarkB200Error):
        model.set_layer(0, bad)
    with pytest.raises(StarkB200Error):
        MoEModel(dict(cfg, head_dim=64), 4)
    model.close()
