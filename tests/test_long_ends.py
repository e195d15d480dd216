"""End rules of the pass queue: last rows at every edge of strips and passes, on either lane of a unit,
ties along the last row and column, values at the s16 clamp, in both lane types."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)
NS = [1, 3, 4, 5, 127, 128, 129, 130, 255, 257, 383, 385, 511, 513, 640, 767, 768, 769, 1025]
FREE = ["first_column_free", "first_row_free", "last_column_free", "last_row_free"]


@pytest.mark.parametrize("ends", ["last_column_free", "last_row_free", "first_column_free,last_column_free",
                                  "first_row_free,last_row_free", "last_column_free,last_row_free",
                                  "first_column_free,first_row_free,last_column_free,last_row_free"])
@pytest.mark.parametrize("scores", [(2, -3, -5, -1), (1, 0, -1, 0), (3, -20, -40, -12)])
@pytest.mark.parametrize("width", [0, 32])
def test_end_rules_equal_oracle(built_lib, oracle, ends, scores, width):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pairwise_aligner_gb300 as pa
    rng = np.random.default_rng(11)
    s1, s2 = [], []
    for k, n in enumerate(NS * 3):
        m = [int(rng.integers(1, 60)), n, int(rng.integers(300, 900))][k % 3]
        b = ACGT[rng.integers(0, 4, n)]
        a = np.resize(b, m) if k % 2 else ACGT[rng.integers(0, 4, m)]
        a = np.where(rng.random(m) < 0.9, a, ACGT[rng.integers(0, 4, m)]).astype(np.uint8)
        if k % 5 == 0:
            a[:] = b[:] = ord("A")                       # ties everywhere
        s1.append(bytes(a))
        s2.append(bytes(b))
    match, mismatch, go, ge = scores
    free = {k: k in ends.split(",") for k in FREE}
    c = dict(local=False, match=match, mismatch=mismatch, gap_open=go, gap_extension=ge, width_hint=width, **free)
    q, qo = pa.pack(s1)
    t, to = pa.pack(s2)
    ctx = pa.Context(0)
    ctx.set_cta_threshold(1)                             # every pair on the queue
    res = pa.Aligner(c, context=ctx).compute_arrays(q, qo, t, to)
    sc, e1, e2 = oracle.align_batch(oracle.make_cfg(match, mismatch, go, ge, **free), q, qo, t, to)
    bad = np.flatnonzero((res["score"] != sc) | (res["end1"] != e1) | (res["end2"] != e2))
    assert len(bad) == 0, (len(bad), [(len(s1[k]), len(s2[k])) for k in bad[:5]], res[bad[:5]],
                           list(zip(sc[bad[:5]], e1[bad[:5]], e2[bad[:5]])))
    ctx.close()


@pytest.mark.parametrize("shape", [(1, 70000), (17, 30000), (100, 3000), (300, 6500), (700, 2900)])
@pytest.mark.parametrize("kw", [dict(), dict(local=True), {k: True for k in FREE}], ids=["global", "local", "free"])
@pytest.mark.parametrize("width", [0, 32])
def test_few_tall_pairs_equal_oracle(built_lib, oracle, shape, kw, width):
    """Few pairs of many more rows than columns: passes of up to 768 rows, whatever the batch's work."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pairwise_aligner_gb300 as pa
    rng = np.random.default_rng(12)
    m, n = shape
    s1, s2 = [], []
    for k in range(3):
        a, b = ACGT[rng.integers(0, 4, m)], ACGT[rng.integers(0, 4, n + k)]
        b[n // 2:n // 2 + m] = a[:len(b[n // 2:n // 2 + m])]
        s1.append(bytes(a))
        s2.append(bytes(b))
    local = bool(kw.get("local"))
    free = {k: local or bool(kw.get(k)) for k in FREE}
    q, qo = pa.pack(s1)
    t, to = pa.pack(s2)
    ctx = pa.Context(0)
    ctx.set_cta_threshold(1)
    c = dict(local=local, match=2, mismatch=-3, gap_open=-5, gap_extension=-1, width_hint=width, **free)
    res = pa.Aligner(c, context=ctx).compute_arrays(q, qo, t, to)
    sc, e1, e2 = oracle.align_batch(oracle.make_cfg(2, -3, -5, -1, local=local, **free), q, qo, t, to)
    assert np.array_equal(res["score"], sc) and np.array_equal(res["end1"], e1) and np.array_equal(res["end2"], e2)
    ctx.close()


def test_long_pairs_after_short_ones_in_the_same_slots(built_lib, oracle):
    """The passes' boundary cells are the slots that short pairs of earlier calls, tracebacks and other
    long pairs have written: alternating calls of one context stay exact."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pairwise_aligner_gb300 as pa
    rng = np.random.default_rng(14)
    ctx = pa.Context(0)

    def batch(shapes):
        s1 = [bytes(ACGT[rng.integers(0, 4, m)]) for m, _ in shapes]
        return (*pa.pack(s1), *pa.pack([bytes(ACGT[rng.integers(0, 4, n)]) for _, n in shapes]))

    for k, width in enumerate((0, 32, 0, 32)):
        for local in (False, True):
            f = dict.fromkeys(FREE, local)
            c = dict(local=local, match=2, mismatch=-3, gap_open=-5, gap_extension=-1, width_hint=width, **f)
            oc = oracle.make_cfg(2, -3, -5, -1, local=local, **f)
            al = pa.Aligner(c, context=ctx)
            for shapes in ([(int(m), 70) for m in rng.integers(1, 200, 400)], [(1200, 1300 + k), (2000, 900)] * 4):
                b = batch(shapes)
                res = al.compute_arrays(*b)
                sc, e1, e2 = oracle.align_batch(oc, *b)
                assert np.array_equal(res["score"], sc) and np.array_equal(res["end1"], e1)
                assert np.array_equal(res["end2"], e2)
            b = batch([(700, 1100)] * 6)
            res = al.compute_traceback_arrays(*b)[0]
            assert np.array_equal(res["score"], oracle.align_batch(oc, *b)[0])
    ctx.close()


@pytest.mark.parametrize("shapes", [[(8300, n) for n in (126, 127, 128, 129, 130)] * 4,
                                    [(m, 2800) for m in (382, 383, 384, 385, 386)] * 4 + [(64, 9000)] * 1020],
                         ids=["flat", "narrow"])
@pytest.mark.parametrize("kw", [dict(), dict(local=True), {k: True for k in FREE}], ids=["global", "local", "free"])
@pytest.mark.parametrize("width", [0, 32])
def test_pairs_on_both_sides_of_the_one_warp_rules(built_lib, oracle, shapes, kw, width):
    """Pairs above the long threshold: up to 128 rows, or 384 columns in a batch full of narrow pairs, they
    stay with the short-pair kernel."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pairwise_aligner_gb300 as pa
    rng = np.random.default_rng(13)
    s1, s2 = [], []
    for m, n in shapes:
        a, b = ACGT[rng.integers(0, 4, m)], ACGT[rng.integers(0, 4, n)]
        w = min(m, n)
        at = int(rng.integers(0, max(m, n) - w + 1))
        if n > m:
            b[at:at + w] = a
        else:
            a[at:at + w] = b
        s1.append(bytes(a))
        s2.append(bytes(b))
    local = bool(kw.get("local"))
    free = {k: local or bool(kw.get(k)) for k in FREE}
    q, qo = pa.pack(s1)
    t, to = pa.pack(s2)
    c = dict(local=local, match=2, mismatch=-3, gap_open=-5, gap_extension=-1, width_hint=width, **free)
    al = pa.Aligner(c, context=pa.Context(0))
    res = al.compute_arrays(q, qo, t, to)
    sc, e1, e2 = oracle.align_batch(oracle.make_cfg(2, -3, -5, -1, local=local, **free), q, qo, t, to)
    assert np.array_equal(res["score"], sc) and np.array_equal(res["end1"], e1) and np.array_equal(res["end2"], e2)
    al.context.close()
