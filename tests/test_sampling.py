"""The stochastic sampler: the oracle against the published Philox4x32-10 known answers and the
reference's own unit-interval test, host-side seed derivation, and (GPU) the device sampler against
the oracle on seeded rows."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from oracle import oracle as O
from stark_b200.engine import position_seed


def test_philox_known_answers():
    """The three known-answer vectors published with the Philox generator (Random123 `kat_vectors`,
    philox4x32 with 10 rounds): zeros, all ones, and the digits of pi."""
    assert O.philox4x32_10([0, 0, 0, 0], [0, 0]).tolist() == [0x6627E8D5, 0xE169C58D, 0xBC57AC4C, 0x9B00DBD8]
    assert O.philox4x32_10([0xFFFFFFFF] * 4, [0xFFFFFFFF] * 2).tolist() == [0x408F276D, 0x41C83B0E, 0xA20BC7C6, 0x6D5451FD]
    assert O.philox4x32_10([0x243F6A88, 0x85A308D3, 0x13198A2E, 0x03707344], [0xA4093822, 0x299F31D0]).tolist() == [
        0xD16CFE09, 0x94FDCCEB, 0x5001E420, 0x24126EA1]


def test_unit_interval_stays_open():
    """crates/stark-engine/unit/encodable_block/sampling/gumbel_test.rs:8-12."""
    assert O.unit_interval(0xFFFFFFFF) == 1.0 - 2.0 ** -24
    assert O.unit_interval(0) == 2.0 ** -24
    assert O.unit_interval(255) == 2.0 ** -24


def test_counter_layout_and_seed_derivation():
    # revidx (gumbel.rs:66-80): 1024 threads, 4 words per counter, vocab rounded up to 4096 per thread
    assert O.revidx(0, 151936) == (0, 0)
    assert O.revidx(1023, 151936) == (1023 * 38, 0)
    assert O.revidx(1024, 151936) == (0, 1)
    assert O.revidx(4096 + 7, 151936) == (7 * 38 + 1, 0)
    for seed, pos in [(0, 0), (1, 2), (2 ** 64 - 1, 5), (123456789, 4096)]:
        assert position_seed(seed, pos) == O.prng_derive(seed, pos)
    assert position_seed(0, 0) == 0  # the finalizer fixes zero


def test_oracle_sampler_semantics():
    rng = np.random.default_rng(0)
    l = rng.standard_normal(1000).astype(np.float32)
    assert O.unified_sampling(l) == int(l.argmax())
    tie = l.copy()
    tie[[10, 700]] = tie.max() + 1
    assert O.unified_sampling(tie) == 10                       # first index of the maximum
    bad = l.copy()
    bad[5] = np.inf
    assert O.unified_sampling(bad) == 0xFFFFFFFF               # non-finite logit: invalid row
    assert O.unified_sampling(l, seed=3, top_k=1) == int(l.argmax())   # one candidate left: noise cannot matter
    order = np.argsort(-l, kind="stable")
    for seed in range(20):
        assert O.unified_sampling(l, seed=seed, top_k=5) in order[:5].tolist()
        assert O.unified_sampling(l, seed=seed, temperature=0.5, min_p=0.5) in np.flatnonzero(
            l / np.float32(0.5) >= (l / np.float32(0.5)).max() + np.log(np.float32(0.5))).tolist()
    draws = {O.unified_sampling(l, seed=s, temperature=1.0) for s in range(64)}
    assert len(draws) > 20                                     # the noise really spreads the choice
    huge = np.array([3e38, 1.0, -3e38], np.float32)            # 1/T overflows the product: centred, not invalid
    assert O.unified_sampling(huge, seed=1, temperature=0.01) == 0


@pytest.mark.gpu
def test_device_sampler_matches_oracle():
    from stark_b200 import ops
    rng = np.random.default_rng(5)
    vocab = 151936
    base = (rng.standard_normal(vocab) * 3.0).astype(np.float32)
    bf = O.bf16_to_f32(O.f32_to_bf16(base))  # bf16-valued logits: many exact ties, as in the engine
    cases = [dict(), dict(seed=11), dict(seed=12, temperature=0.7), dict(seed=13, temperature=0.8, top_k=40),
             dict(seed=14, temperature=1.3, top_p=0.9), dict(seed=15, min_p=0.05),
             dict(seed=16, temperature=0.6, top_k=50, top_p=0.95, min_p=0.02), dict(top_k=3), dict(seed=17, top_k=1)]
    agree = 0
    for i, kw in enumerate(cases):
        for row in (base, bf):
            want = O.unified_sampling(row, **kw)
            got = ops.sample(row, **kw)
            agree += int(got == want)
    # device expf / logf differ from the host libm in the last bit, which can flip a near-tie of noisy scores
    assert agree >= 2 * len(cases) - 1, agree
    assert ops.sample(O.f32_to_bf16(bf), seed=21, temperature=0.9, top_k=20) == O.unified_sampling(
        bf, seed=21, temperature=0.9, top_k=20)               # bf16 input
    bad = base.copy()
    bad[77] = np.nan
    assert ops.sample(bad, seed=1) == 0xFFFFFFFF
    from stark_b200._lib import StarkB200Error
    for kw in (dict(temperature=0.0), dict(temperature=101.0), dict(top_k=0), dict(top_k=vocab + 1), dict(top_p=0.0),
               dict(top_p=1.5), dict(min_p=-0.1)):
        with pytest.raises(StarkB200Error):
            ops.sample(base, seed=1, **kw)
    small = rng.standard_normal(1000).astype(np.float32)      # a short row: idle lanes in the sort
    for s in range(8):
        assert ops.sample(small, seed=s, temperature=0.7, top_k=10, top_p=0.9) == O.unified_sampling(
            small, seed=s, temperature=0.7, top_k=10, top_p=0.9)


def _awkward_row(kind, vocab, rng):
    if kind == "equal":          # every partial sum is a whole number, every quotient the same
        return np.zeros(vocab, np.float32)
    if kind == "few":            # long runs of equal terms: half way between two sums again and again
        return rng.choice(np.array([0.0, -0.0, 0.6931472, 1.3862944, -2.0794415], np.float32), vocab)
    row = (rng.standard_normal(vocab) * 3.0).astype(np.float32)
    if kind == "peaked":         # the tail stops moving the sums early
        row[vocab // 2] = 40.0
    if kind == "subnormal":      # scaling merges values that the logits tell apart
        row = (row * np.float32(1e-39)).astype(np.float32)
    if kind == "huge":           # scaling overflows: centred
        row = row * np.float32(2e37)  # finite at five standard deviations
    return O.bf16_to_f32(O.f32_to_bf16(row))


AWKWARD_SETTINGS = [
    (1, dict(top_p=0.5)), (2, dict(temperature=0.7, top_k=20, top_p=0.95)), (3, dict(temperature=1.7, top_p=1.0)), (4, dict(min_p=0.3)),
    (5, dict(temperature=0.01, top_p=0.999, min_p=0.001)), (6, dict(temperature=0.9)), (7, dict(top_k=5461))]


@pytest.mark.gpu
@pytest.mark.parametrize("seed,setting", AWKWARD_SETTINGS)
def test_device_sampler_on_awkward_rows(seed, setting):
    """Rows shorter than the cluster, at the borders of a stretch of the sums, with ties, merged and centred values; as f32
    and as bf16 (two sorting passes instead of four)."""
    from stark_b200 import ops
    misses = []
    for kind in ("equal", "few", "normal", "peaked", "subnormal", "huge"):
        for vocab in (1, 15, 257, 1023, 8192, 8193, 16385, 151936):
            row = _awkward_row(kind, vocab, np.random.default_rng([vocab, len(kind)]))
            kw = dict(setting, **({"top_k": min(setting["top_k"], vocab)} if "top_k" in setting else {}))
            want = O.unified_sampling(row, seed=seed, **kw)
            misses += [(kind, vocab) for given in (row, O.f32_to_bf16(row)) if ops.sample(given, seed=seed, **kw) != want]
    # Device and host expf / logf differ by an ulp or two: scores within 1e-6 of each other can change places, and a cut in a flat
    # row of V terms can move by V * 1e-7 * V / 2 of them.  Either decides a pick about once in ten thousand of these.
    assert len(misses) <= 1, misses


def _gumbel(seed, index, vocab):
    return O.gumbel_float(seed, *O.revidx(int(index), vocab))


def _cut_row(vocab, half):
    """60 candidates a few per cent of the mass each, in scrambled places, over a tail that takes half of the sum."""
    rng = np.random.default_rng(vocab)
    row = (np.log(60.0 * 0.5 / max(vocab - 60, 1)) - 1.5 + 0.3 * rng.standard_normal(vocab)).astype(np.float32)
    places = rng.permutation(vocab)[:60]
    row[places] = np.linspace(0.0, -0.9375, 61)[:60].astype(np.float32)  # 1 / 64 apart: bf16 tells them apart
    return O.bf16_to_f32(O.f32_to_bf16(row)) if half else row


def _picks(row, order, kept, seeds):
    """For every seed the rank that wins among the first `kept`, by noise of the oracle's generator; near-ties left out."""
    out = {}
    for seed in seeds:
        scores = sorted(((float(row[order[n]]) + _gumbel(seed, order[n], row.size), n) for n in range(kept)), reverse=True)
        if len(scores) == 1 or scores[0][0] - scores[1][0] > 1e-3:
            out[seed] = scores[0][1]
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("vocab", [64, 8193, 40000, 151936])
@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("kept", [1, 2, 7, 33])
def test_device_sampler_cuts_where_the_sums_say(vocab, half, kept):
    """A threshold half way between two partial sums keeps exactly the candidates below it: seeds whose noise favours the last
    one kept pick it, and seeds whose noise favours the first one cut do not.  Rows whose norm has many stretches of terms."""
    from stark_b200 import ops
    row = _cut_row(vocab, half)
    order = np.argsort(-row, kind="stable")
    terms = np.exp((row[order] - row[order[0]]).astype(np.float64))
    mass = np.cumsum(terms) / terms.sum()
    top_p = float((mass[kept - 2] + mass[kept - 1]) / 2 if kept > 1 else mass[0] / 2)
    min_p = float((terms[kept - 1] + terms[kept]) / 2)
    given = O.f32_to_bf16(row) if half else row
    inside = [(seed, n) for seed, n in _picks(row, order, kept, range(200)).items() if n == kept - 1][:4]
    wider = [seed for seed, n in _picks(row, order, kept + 1, range(200)).items() if n == kept][:4]
    assert inside and wider
    for setting in (dict(top_p=top_p), dict(min_p=min_p), dict(top_k=kept), dict(top_p=top_p, top_k=kept + 5), dict(top_p=0.999, min_p=min_p)):
        for seed, n in inside:
            assert ops.sample(given, seed=seed, **setting) == order[n] == O.unified_sampling(row, seed=seed, **setting), (setting, seed)
        within = _picks(row, order, kept, wider)
        for seed in within:
            assert ops.sample(given, seed=seed, **setting) == order[within[seed]] == O.unified_sampling(row, seed=seed, **setting), (setting, seed)


CLUSTER_FIT = """
#include "cluster_fit.cuh"
#include <cstdio>
using namespace sb;
// A runtime of three devices: 0 and 2 hold clusters of 16 of a kernel opted in there, 1 does not.
static int current = 0, opted[3][2], queries = 0, errors = 0;
static int kernels[2];
static int which(const void *f) { return f == &kernels[1]; }
extern "C" cudaError_t cudaGetDevice(int *d) { *d = current; return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { ++errors; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
    opted[current][which(f)] += a == cudaFuncAttributeNonPortableClusterSizeAllowed && v == 1;
    return cudaSuccess;
}
extern "C" cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *f, const cudaLaunchConfig_t *c) {
    ++queries;
    *n = current != 1 && opted[current][which(f)] && c->gridDim.x == 16 && c->numAttrs == 1 && c->attrs->val.clusterDim.x == 16;
    return current == 1 ? cudaErrorInvalidClusterSize : cudaSuccess;
}
int main() {
    static ClusterFit known[2];
    for (int round = 0; round < 2; ++round)
        for (current = 0; current < 3; ++current)
            for (int k = 0; k < 2; ++k) std::printf("%u ", cluster_fit(&kernels[k], cudaLaunchConfig_t{}, known[k]));
    std::printf("| %d %d %d %d %d", queries, errors, opted[0][0], opted[1][1], opted[2][0]);
}
"""


def test_cluster_size_is_known_per_device(tmp_path):
    """What one device allows says nothing about another: every device is opted in and asked once, for each kernel."""
    src, exe = tmp_path / "fit.cpp", tmp_path / "fit"
    src.write_text(CLUSTER_FIT)
    root = Path(__file__).resolve().parents[1]
    subprocess.run(["g++", "-std=c++17", f"-I{root / 'stark_b200' / 'csrc'}", "-I/usr/local/cuda/include", str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out == "16 16 8 8 16 16 " * 2 + "| 6 2 1 1 1", out


@pytest.mark.gpu
def test_sampler_on_two_devices():
    from stark_b200 import _lib, ops
    if ops.device_count() < 2:
        pytest.skip("needs two GPUs")
    row = np.random.default_rng(4).standard_normal(9000).astype(np.float32)
    for ordered in (False, True):
        seen = []
        for device in (0, 1, 0):
            _lib.check(_lib.load().stark_b200_set_device(device), "set_device")
            seen.append(ops.sample(row, seed=11, temperature=0.8, top_k=40, ordered=ordered))
        assert len(set(seen)) == 1


@pytest.mark.gpu
def test_model_sampling_follows_the_last_row():
    from stark_b200 import synthetic as S
    from stark_b200.engine import DenseModel
    cfg = S.CONFIGS["tiny"]
    model = DenseModel.load(cfg, S.dense_weights(cfg, seed=0), context_tokens=64)
    model.prefill(S.prompt(cfg, 9, seed=1))
    logits = model.logits()
    assert model.sample() == model.argmax() == O.unified_sampling(logits)
    for pos in range(4):
        seed = position_seed(42, model.position)
        tok = model.sample(seed=seed, temperature=0.8, top_k=20)
        assert tok == O.unified_sampling(model.logits(), seed=seed, temperature=0.8, top_k=20)
        model.step_async(tok)


# ---- the generation worker's host sampler (sorted f64 probabilities, SplitMix64) ----

def _full_sort_sample(logits, rng, temperature, top_k=None, top_p=None, min_p=None):
    """An independent restatement in numpy/Python of the full-sort form of the sampler
    (crates/stark-generate/src/hybrid.rs:1773-1816 keeps the same form as its differential oracle)."""
    import math
    logits = np.asarray(logits, np.float32)
    order = sorted(range(logits.size), key=lambda i: (O.descending_sample_key(float(logits[i])), i))
    order = order[:min(top_k, logits.size) if top_k is not None else logits.size]
    top = logits[order[0]]
    p = [math.exp(float(np.float32(np.float32(logits[i] - top) / np.float32(temperature)))) for i in order]
    total = 0.0
    for v in p:
        total += v
    kept, cum = 0, 0.0
    for v in p:
        if kept > 0 and ((min_p is not None and v < float(np.float32(min_p)))
                         or (top_p is not None and cum / total >= float(np.float32(top_p)))):
            break
        cum += v
        kept += 1
    u, rng = O.splitmix64_uniform(rng)
    target, mass = u * cum, 0.0
    for n in range(kept):
        mass += p[n]
        if target < mass:
            return order[n], rng
    return order[kept - 1], rng


def test_splitmix64_known_answers():
    """The first outputs of SplitMix64 from state 0 (the vectors published with the generator), seen
    through `uniform` (hybrid.rs:1103-1111): the top 53 bits scaled by 2^-53, state advanced by the step."""
    state = 0
    for word in (0xE220A8397B1DCDAF, 0x6E789E6AA1B965F4, 0x06C45D188009454F):
        u, state = O.splitmix64_uniform(state)
        assert u == (word >> 11) / 2.0 ** 53
    assert state == (3 * O.SPLITMIX64_STEP) % 2 ** 64


def test_host_sampler_reference_cases():
    """hybrid.rs:1653-1664, 1751-1769, 2032-2062 (the cases the reference's own tests assert) and the
    descending key's order (hybrid.rs:1320-1328)."""
    f = lambda *v: np.array(v, np.float32)
    assert O.host_sampling(f(-1000.0, 1000.0), 99, 1.0, top_k=1, top_p=0.5)[0] == 1
    for seed in range(100):
        assert O.host_sampling(f(0.0, -1.0), seed, 1.0, min_p=0.9)[0] == 0   # min-p is relative to the top one
    assert O.host_sampling(f(0.0, 0.0), 12) == O.host_sampling(f(0.0, 0.0), 12)
    for bad in (np.nan, np.inf, -np.inf):
        assert O.host_sampling(f(0.0, bad), 0) == (0xFFFFFFFF, 0)             # no draw: the state stays
    assert O.host_sampling(f(), 0)[0] == 0xFFFFFFFF
    keys = [O.descending_sample_key(v) for v in (np.inf, 3.0, 1e-45, 0.0, -0.0, -1e-45, -3.0, -np.inf)]
    assert keys == sorted(keys) and len(set(keys)) == len(keys)              # +0 sorts before -0
    tok, state = O.host_sampling(f(0.5, 0.25), 7)
    assert state == (7 + O.SPLITMIX64_STEP) % 2 ** 64


def test_host_sampler_matches_full_sort_form():
    rng = np.random.default_rng(31)
    for n in (1, 2, 33, 257, 2000):
        row = (rng.standard_normal(n) * 2.5).astype(np.float32)
        row[rng.integers(0, n, max(1, n // 8))] = row[0]                      # ties
        if n > 2:
            row[1], row[2] = 0.0, -0.0
        for kw in (dict(), dict(top_k=5), dict(top_p=0.8), dict(min_p=0.1), dict(top_k=40, top_p=0.95, min_p=0.01)):
            for seed in (0, 1, 2 ** 63 + 5):
                for t in (0.5, 1.0, 1.7):
                    assert O.host_sampling(row, seed, t, **kw) == _full_sort_sample(row, seed, t, **kw)


@pytest.mark.gpu
def test_device_ordered_sampler_matches_oracle():
    from stark_b200 import ops
    from stark_b200._lib import StarkB200Error
    rng = np.random.default_rng(6)
    vocab = 151936
    base = (rng.standard_normal(vocab) * 3.0).astype(np.float32)
    bf = O.bf16_to_f32(O.f32_to_bf16(base))
    peaked = base.copy()
    peaked[4242] = 60.0                                                       # the tail stops moving the sums early
    cases = [dict(), dict(temperature=0.7), dict(temperature=0.8, top_k=40), dict(temperature=1.3, top_p=0.9),
             dict(min_p=0.05), dict(temperature=0.6, top_k=50, top_p=0.95, min_p=0.02), dict(top_k=1),
             dict(top_p=1.0), dict(temperature=100.0, top_p=0.999), dict(temperature=0.05)]
    total = agree = 0
    for kw in cases:
        for row in (base, bf, peaked):
            for seed in (3, 2 ** 64 - 1, 0x1234_5678_9ABC_DEF0):
                want, _ = O.host_sampling(row, seed, kw.get("temperature", 1.0),
                                          **{k: v for k, v in kw.items() if k != "temperature"})
                got = ops.sample(row, seed=seed, ordered=True, **kw)
                total += 1
                agree += int(got == want)
    # the device's f64 exp is within 1 ulp of the host's, not identical: a target that lands within a few
    # ulps of a partial sum can resolve to the neighbouring candidate
    assert agree >= total - 2, (agree, total)
    assert ops.sample(O.f32_to_bf16(bf), seed=21, temperature=0.9, top_k=20, ordered=True) == O.host_sampling(
        bf, 21, 0.9, top_k=20)[0]                                             # bf16 input
    bad = base.copy()
    bad[77] = -np.inf
    assert ops.sample(bad, seed=1, ordered=True) == 0xFFFFFFFF
    with pytest.raises(StarkB200Error):
        ops.sample(base, ordered=True)                                        # the ordered sampler only draws
    zeros = np.zeros(70, np.float32)
    zeros[1::2] = -0.0                                                        # +0 candidates come first, by id
    small = rng.standard_normal(1000).astype(np.float32)
    for s in range(8):
        assert ops.sample(zeros, seed=s, top_k=35, ordered=True) == O.host_sampling(zeros, s, top_k=35)[0]
        assert ops.sample(zeros, seed=s, top_k=35, ordered=True) % 2 == 0
        assert ops.sample(small, seed=s, temperature=0.7, top_k=10, top_p=0.9, ordered=True) == O.host_sampling(
            small, s, 0.7, top_k=10, top_p=0.9)[0]
