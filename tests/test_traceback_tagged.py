"""Traceback with tagged values: row counts at the edges of strips, words and passes, every end-gap
rule, tables, bytes (N among the rows, positive mismatch) and matrices, ties (unit scores), and
scores on both sides of the 26-bit line, byte for byte against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NS = [1, 2, 31, 63, 64, 65, 128, 255, 256, 257, 320, 511, 512, 513, 576, 769, 1025]
MODES = [dict(), dict(local=True), dict(first_column_free=True, last_column_free=True),
         dict(first_row_free=True, last_row_free=True), dict(last_row_free=True, last_column_free=True)]
ACGT = np.frombuffer(b"ACGT", np.uint8)


def _batch(pa, seed, alphabet):
    rng = np.random.default_rng(seed)
    s1, s2 = [], []
    for k, n in enumerate(NS * 2 + [0, 5]):
        m = int(rng.integers(1, 90)) if k % 3 else max(1, n + int(rng.integers(-3, 4)))
        if k == 2 * len(NS) + 1:
            m = 0
        b = alphabet[rng.integers(0, len(alphabet), n)]
        a = alphabet[rng.integers(0, len(alphabet), m)]
        w = min(m, n)
        a[:w] = np.where(rng.random(w) < 0.85, b[:w], a[:w])
        if w > 20:                                     # a gap of a few symbols
            a = np.concatenate([a[:w // 2], a[w // 2 + 4:]])
        s1.append(bytes(a))
        s2.append(bytes(b))
    return s1, s2


@pytest.mark.parametrize("kw", MODES, ids=["global", "local", "free_column", "free_row", "free_end"])
@pytest.mark.parametrize("scores", [(2, -3, -5, -1), (1, -1, 0, -1), (1, 0, -1, 0), (2, 1, -3, -1), (60000, -50000, -30000, -9000),
                                    (120, -120, -90, -40)])
@pytest.mark.parametrize("kind", ["dna", "n", "matrix"])
def test_paths_equal_oracle(built_lib, oracle, kw, scores, kind):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pairwise_aligner_gb300 as pa
    match, mismatch, go, ge = scores
    local = bool(kw.get("local"))
    alphabet = ACGT if kind == "dna" else np.frombuffer(b"ACGTNa", np.uint8)
    c = dict(local=local, match=match, mismatch=mismatch, gap_open=go, gap_extension=ge, first_column_free=local,
             first_row_free=local, last_column_free=local, last_row_free=local)
    c.update(kw)
    free = {k: c[k] for k in ("first_column_free", "first_row_free", "last_column_free", "last_row_free")}
    if kind == "matrix":
        sc = np.full((6, 6), mismatch)
        np.fill_diagonal(sc, match)
        c["matrix"] = (bytes(alphabet), [int(x) for x in sc.ravel()])
        oc = oracle.make_cfg(0, 0, go, ge, local=local, matrix=c["matrix"], **free)
    else:
        oc = oracle.make_cfg(match, mismatch, go, ge, local=local, **free)
    s1, s2 = _batch(pa, 7, alphabet)
    ctx = pa.Context(0)
    for x, a, b in zip(pa.Aligner(c, context=ctx).compute_traceback(s1, s2), s1, s2):
        want = oracle.traceback(oc, a, b)
        assert (x.score(), *x.begin_position(), *x.end_position(), x.ops()) == want, (len(a), len(b))
    ctx.close()
