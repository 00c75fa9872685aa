"""GPU parity of the quantized matvec against the CPU oracle, through the C ABI."""
import numpy as np
import pytest

from oracle import oracle as O
from stark_b200 import synthetic as S

pytestmark = pytest.mark.gpu

# per-op bar: integer unpack bit-exact; outputs within 1e-2 relative (bf16 in, f32 accumulate)
REL_TOL = 1e-2


def _rel_err(got_bits, want_bits):
    got, want = O.bf16_to_f32(got_bits).astype(np.float64), O.bf16_to_f32(want_bits).astype(np.float64)
    scale = np.maximum(np.abs(want), np.abs(want).mean())
    return np.abs(got - want) / scale


@pytest.mark.parametrize("rows,columns", [(16, 64), (48, 128), (4096, 4096), (1000, 1024), (6144, 4096),
                                          (4096, 12288)])
def test_unpack_is_bit_exact(rows, columns):
    from stark_b200.ops import QMatrix
    w = S.matvec_case(seed=rows + columns, rows=rows, columns=columns)
    q = QMatrix.from_affine(w["codes"], w["scales"], w["biases"], rows, columns)
    want = O.unpack_codes(w["codes"], 4, rows * columns).reshape(rows, columns)
    assert np.array_equal(q.unpack_codes(), want)
    assert q.device_bytes() == ((rows + 15) // 16) * (columns // 64) * 576


@pytest.mark.parametrize("rows,columns", [(16, 64), (48, 128), (4096, 4096), (1000, 1024), (6144, 4096),
                                          (4096, 12288), (151936, 1024)])
def test_matvec_bf16_matches_oracle(rows, columns):
    from stark_b200.ops import QMatrix, take_device_error
    w = S.matvec_case(seed=7 + rows, rows=rows, columns=columns)
    q = QMatrix.from_affine(w["codes"], w["scales"], w["biases"], rows, columns)
    got = q.matvec(w["x"])
    assert take_device_error() == 0
    want = O.affine_matvec_bf16(w["codes"], w["scales"], w["biases"], w["x"], rows, columns,
                                threads=O.max_threads())[0]
    err = _rel_err(got, want)
    assert err.max() < REL_TOL
    # far tighter in practice: same products, f32 accumulation in a different order
    assert (got != want).mean() < 0.02


@pytest.mark.parametrize("rows,columns", [(16, 64), (40, 192), (1000, 1024), (1760, 4096), (9472, 576), (1024, 3072), (2080, 448)])
def test_matrices_requested_whole(rows, columns):
    """Fewer column groups than warps, ragged slices, a last row tile in part, the widest row and the most tiles, plain (up
    to 148 tiles) and gated, against the streaming kernel: the same products, f32 sums formed in another order, one rounding to bf16."""
    from stark_b200 import _lib
    from stark_b200.ops import QMatrix, qmv_swiglu, take_device_error
    w = S.matvec_case(seed=5 + rows, rows=rows, columns=columns)
    make = lambda pair: QMatrix.from_affine(w["codes"], w["scales"], w["biases"], rows, columns, pair_halves=pair)  # noqa: E731
    plain, pair = make(False), make(True) if rows % 32 == 0 else None
    seen = []
    try:
        for short in (0, 1):
            _lib.check(_lib.load().stark_b200_set_tunable(b"qmv_short", short), "set_tunable")
            seen.append((plain.matvec(w["x"]), qmv_swiglu(pair, w["x"]) if pair else None))
    finally:
        _lib.check(_lib.load().stark_b200_set_tunable(b"qmv_short", 1), "set_tunable")
    assert take_device_error() == 0
    for streamed, whole in zip(*seen):
        if streamed is None:
            continue
        assert (streamed != whole).mean() < 0.02
        assert _rel_err(whole, streamed).max() <= 3 * 2.0 ** -7  # a unit of the last place; of both factors and their product


@pytest.mark.parametrize("hidden,inter", [(64, 64), (192, 448), (576, 64), (1024, 1216), (4096, 320)])
def test_matrices_requested_whole_with_norm_and_residual(hidden, inter):
    """The forms that only a token uses -- the norm in the prologue (fewer column groups than warps, ragged slices, the widest
    row), the residual in the epilogue -- through one layer, against the streaming kernel and the oracle."""
    from stark_b200 import _lib
    from stark_b200.engine import DenseModel
    from stark_b200.ops import take_device_error
    from tests.test_model_gpu import assert_logits_accepted
    cfg = dict(S.CONFIGS["tiny"], layers=1, hidden=hidden, inter=inter, q_heads=2, kv_heads=1, vocab=512)
    w = S.dense_weights(cfg, seed=hidden, zero_point=7.5)
    ids, seen = S.prompt(cfg, 3, seed=4), []
    try:
        for short in (0, 1):
            _lib.check(_lib.load().stark_b200_set_tunable(b"qmv_short", short), "set_tunable")
            model = DenseModel.load(cfg, w, context_tokens=16)
            seen.append([O.f32_to_bf16(model.step(int(t))) for t in ids])
            model.close()
    finally:
        _lib.check(_lib.load().stark_b200_set_tunable(b"qmv_short", 1), "set_tunable")
    assert take_device_error() == 0
    oracle = O.DenseOracle(cfg, w, capacity=16)
    for t, streamed, whole in zip(ids, *seen):
        assert_logits_accepted(streamed, whole)
        assert_logits_accepted(oracle.step(int(t)), whole)


def test_matvec_group_output_plane_layout():
    from stark_b200.ops import QMatrix
    rows, columns = 100, 256
    w = S.matvec_case(seed=11, rows=rows, columns=columns)
    pitch = (rows + 3) // 4 * 4
    st = np.zeros((columns // 64, pitch), np.uint16)
    bt = np.zeros((columns // 64, pitch), np.uint16)
    st[:, :rows] = w["scales"].T
    bt[:, :rows] = w["biases"].T
    q = QMatrix.from_affine(w["codes"], st, bt, rows, columns, scale_layout=1, plane_pitch=pitch)
    want = O.affine_matvec_bf16(w["codes"], w["scales"], w["biases"], w["x"], rows, columns)[0]
    assert _rel_err(q.matvec(w["x"]), want).max() < REL_TOL


def test_matvec_f32_hybrid_conventions():
    from stark_b200._lib import F32
    from stark_b200.ops import QMatrix
    rows, columns = 512, 2048
    w = S.matvec_case(seed=13, rows=rows, columns=columns)
    x = np.random.default_rng(2).standard_normal(columns).astype(np.float32)
    q = QMatrix.from_affine(w["codes"], w["scales"], w["biases"], rows, columns)
    got = q.matvec(x, io_type=F32)
    want = O.affine_matvec_f32(w["codes"], w["scales"], w["biases"], 30, x, rows, columns)
    # the reference's own bound for this comparison: 2e-5 * sum |w x| (weights.rs:4218-4297)
    wf = np.stack([O.affine_row_f32(w["codes"], w["scales"], w["biases"], 30, r, columns) for r in range(rows)])
    bound = 2e-5 * (np.abs(wf) * np.abs(x)).sum(axis=1)
    assert np.all(np.abs(got - want) <= bound)


def test_linearity_and_scaling_at_full_size():
    """Size-independent properties at the 4096x4096 benchmark size."""
    from stark_b200._lib import F32
    from stark_b200.ops import QMatrix
    w = S.matvec_case(seed=0)
    q = QMatrix.from_affine(w["codes"], w["scales"], w["biases"], 4096, 4096)
    rng = np.random.default_rng(4)
    a = rng.standard_normal(4096).astype(np.float32)
    b = rng.standard_normal(4096).astype(np.float32)
    ya, yb, yab = q.matvec(a, io_type=F32), q.matvec(b, io_type=F32), q.matvec(a + b, io_type=F32)
    np.testing.assert_allclose(yab, ya + yb, rtol=0, atol=2e-4 * np.abs(ya).mean() + 1e-4)
    # exact power-of-two scaling of the input scales the output exactly (the kernel rescales by 2^k)
    y4 = q.matvec(O.f32_to_bf16(O.bf16_to_f32(w["x"]) * 4.0))
    y1 = q.matvec(w["x"])
    assert np.array_equal(O.bf16_to_f32(y4), O.bf16_to_f32(y1) * 4.0)
    # zero input -> sum(bias * 0) = 0 exactly
    assert not q.matvec(np.zeros(4096, np.uint16)).any()


def test_repeatability_bitwise():
    from stark_b200.ops import QMatrix
    w = S.matvec_case(seed=21, rows=2048, columns=4096)
    q = QMatrix.from_affine(w["codes"], w["scales"], w["biases"], 2048, 4096)
    first = q.matvec(w["x"])
    for _ in range(3):
        assert np.array_equal(q.matvec(w["x"]), first)


def test_invalid_arguments_are_rejected():
    from stark_b200._lib import StarkB200Error
    from stark_b200.ops import QMatrix
    w = S.matvec_case(seed=1, rows=16, columns=64)
    with pytest.raises(ValueError):
        QMatrix.from_affine(w["codes"], w["scales"], w["biases"], 16, 128)
    q = QMatrix.from_affine(w["codes"], w["scales"], w["biases"], 16, 64)
    with pytest.raises(ValueError):
        q.matvec(np.zeros(63, np.uint16))
    with pytest.raises(StarkB200Error):
        QMatrix.from_affine(w["codes"], w["scales"], w["biases"], 16, 64, group=32)


@pytest.mark.parametrize("rows,columns", [(16, 1024), (1000, 2048), (4800, 3072), (6144, 4096), (100, 8192), (2048, 12288), (9488, 5120)])
def test_column_slices(rows, columns):
    """Warps that own slices of the columns (two to eight groups of 64, one to three chunks), against the shared ring: one row plain and
    gated, two to eight rows with and without the norm.  A last row tile in part, fewer tiles than CTAs, more than a round of them.  The
    same products up to an offset the group sums take out again, f32 sums formed in another order, one rounding to bf16; and no further
    from the 64-bit result."""
    from stark_b200 import _lib
    from stark_b200.ops import QMatrix, qmv_swiglu, take_device_error
    w = S.matvec_case(seed=9 + rows, rows=rows, columns=columns)
    make = lambda pair: QMatrix.from_affine(w["codes"], w["scales"], w["biases"], rows, columns, pair_halves=pair)  # noqa: E731
    plain, pair = make(False), make(True) if rows % 32 == 0 else None
    rng = np.random.default_rng(rows)
    several = {m: S.bf16_normal(rng, m * columns).reshape(m, columns) for m in (2, 5, 8) if m * columns <= 8 * 8192}  # more: refused
    weight = (1.0 + 0.1 * rng.standard_normal(columns)).astype(np.float32)
    seen = []
    try:
        _lib.check(_lib.load().stark_b200_set_tunable(b"qmv_short", 0), "set_tunable")
        for sliced in (0, 1):
            _lib.check(_lib.load().stark_b200_set_tunable(b"qmv_slice", sliced), "set_tunable")
            out = [plain.matvec(w["x"]), qmv_swiglu(pair, w["x"]) if pair else None]
            for m, x in several.items():
                out.append(plain.matvec_rows(x))
                if columns <= 4096:
                    out.append(plain.matvec_rows(x, norm_weight=weight))
                    out.append(plain.matvec_rows(x, epilogue=1, residual=S.bf16_normal(np.random.default_rng(m), m * rows).reshape(m, rows)))
                    if pair:
                        out.append(pair.matvec_rows(x, epilogue=2, norm_weight=weight))
            seen.append(out)
    finally:
        _lib.check(_lib.load().stark_b200_set_tunable(b"qmv_short", 1), "set_tunable")
        _lib.check(_lib.load().stark_b200_set_tunable(b"qmv_slice", 1), "set_tunable")
    assert take_device_error() == 0
    for ring, sliced in zip(*seen):
        if ring is None:
            continue
        assert (ring != sliced).mean() < 0.02
        assert _rel_err(sliced, ring).max() <= 3 * 2.0 ** -7  # a unit of the last place; of both factors and their product
    codes = O.unpack_codes(w["codes"], 4, rows * columns).reshape(rows, columns // 64, 64).astype(np.float64)
    scale, bias = (O.bf16_to_f32(w[k]).astype(np.float64).reshape(rows, -1, 1) for k in ("scales", "biases"))
    exact = (codes * scale + bias).reshape(rows, columns) @ O.bf16_to_f32(w["x"]).astype(np.float64)
    off = [np.linalg.norm(O.bf16_to_f32(out[0]).astype(np.float64) - exact) for out in seen]
    assert off[1] <= 1.02 * off[0]   # rounding to bf16 is the error: the few results that round the other way move it this much
