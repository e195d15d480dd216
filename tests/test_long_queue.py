"""Long pairs on the pass queue: every pair of every batch is sent there (threshold 1) and
compared with the oracle, over the rows per thread that the batch's work selects (4 to 24), the
edges of the passes and of their last chunk, and both lane widths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", dtype=np.uint8)
FREE = dict(first_column_free=True, last_column_free=True, last_row_free=True)
# rows of sequence2 at the edges of passes (multiples of 128 up to 768 rows)
EDGES = [1, 31, 127, 128, 129, 255, 256, 257, 511, 513, 767, 768, 769, 1025, 1537]


@pytest.fixture(scope="module")
def pa(built_lib):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pairwise_aligner_gb300 as pa
    return pa


def _batch(pa, seed, n_pairs):
    """Edge pairs with sequence1 lengths around the 16-column stages, then short filler pairs up to
    n_pairs; half of them related."""
    rng = np.random.default_rng(seed)
    s1, s2 = [], []
    for k in range(n_pairs):
        n = EDGES[k] if k < len(EDGES) else int(rng.integers(1, 60))
        m = (15, 16, 17, 33)[k % 4] if k < 8 else int(rng.integers(1, 90))
        b = ACGT[rng.integers(0, 4, n)]
        a = ACGT[rng.integers(0, 4, m)]
        if k % 2:
            w = min(m, n)
            a[:w] = b[:w]
            a[rng.random(m) < 0.1] = ord("A")
        s1.append(bytes(a))
        s2.append(bytes(b))
    return pa.pack(s1) + pa.pack(s2)


@pytest.mark.parametrize("n_pairs", [15, 3000, 20000])
@pytest.mark.parametrize("width", [0, 32])
@pytest.mark.parametrize("kw", [dict(), dict(local=True), FREE], ids=["global", "local", "free"])
def test_pass_queue_equals_oracle(pa, oracle, n_pairs, width, kw):
    local = bool(kw.get("local"))
    c = dict(local=local, match=2, mismatch=-3, gap_open=-5, gap_extension=-1, first_column_free=local,
             first_row_free=local, last_column_free=local, last_row_free=local, width_hint=width)
    c.update(kw)
    q, qo, t, to = _batch(pa, 100 + n_pairs, n_pairs)
    ctx = pa.Context(0)
    ctx.set_cta_threshold(1)
    al = pa.Aligner(c, context=ctx)
    oc = oracle.make_cfg(2, -3, -5, -1, local=local, first_column_free=c["first_column_free"],
                         first_row_free=c["first_row_free"], last_column_free=c["last_column_free"],
                         last_row_free=c["last_row_free"])
    want = oracle.align_batch(oc, q, qo, t, to)
    for _ in range(2):                               # the second call replays the first one's graph
        res = al.compute_arrays(q, qo, t, to)
        for got, exp in zip((res["score"], res["end1"], res["end2"]), want):
            assert np.array_equal(got, exp)
    ctx.close()
