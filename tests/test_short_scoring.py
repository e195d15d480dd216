"""The short-pair kernel's s32 scorings against the oracle: int8 profiles of a substitution
matrix (symbol counts around the rounding to 4, scores at the limits of a signed byte and one past
them, which leaves the profile path), raw byte comparison, and tables; every group size, on row
counts at the edges of strips, passes and groups without a pair."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 40), (40, 1), (17, 63), (33, 64), (64, 65), (90, 127), (61, 128), (129, 129), (200, 255),
          (77, 256), (150, 257), (300, 511), (40, 513), (5, 700)]
MODES = [dict(), dict(local=True), dict(first_column_free=True, last_column_free=True),
         dict(first_row_free=True, last_row_free=True)]


@pytest.fixture(scope="module")
def pa(built_lib):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pairwise_aligner_gb300 as pa
    return pa


def _batch(pa, seed, alphabet):
    rng = np.random.default_rng(seed)
    s1, s2 = [], []
    for m, n in SHAPES * 3:
        a, b = alphabet[rng.integers(0, len(alphabet), m)], alphabet[rng.integers(0, len(alphabet), n)]
        w = min(m, n)
        if rng.random() < 0.6:
            b[:w] = np.where(rng.random(w) < 0.8, a[:w], b[:w])
        s1.append(bytes(a))
        s2.append(bytes(b))
    return pa.pack(s1) + pa.pack(s2)


def _run(pa, oracle, batch, group, kw, matrix=None, width=0, match=0, mismatch=0):
    local = bool(kw.get("local"))
    c = dict(local=local, match=match, mismatch=mismatch, gap_open=-7, gap_extension=-2, first_column_free=local,
             first_row_free=local, last_column_free=local, last_row_free=local, width_hint=width)
    c.update(kw)
    free = {k: c[k] for k in ("first_column_free", "first_row_free", "last_column_free", "last_row_free")}
    if matrix:
        c["matrix"] = matrix
        oc = oracle.make_cfg(0, 0, -7, -2, local=local, matrix=matrix, **free)
    else:
        oc = oracle.make_cfg(match, mismatch, -7, -2, local=local, **free)
    ctx = pa.Context(0, group_threads=group)
    res = pa.Aligner(c, context=ctx).compute_arrays(*batch)
    ctx.close()
    for got, want in zip((res["score"], res["end1"], res["end2"]), oracle.align_batch(oc, *batch)):
        assert np.array_equal(got, want)
    assert (res["width"] == 32).all()


@pytest.mark.parametrize("kw", MODES, ids=["global", "local", "free_column", "free_row"])
@pytest.mark.parametrize("group", [0, 4, 8, 16, 32])
@pytest.mark.parametrize("dim,hi,lo", [(1, 5, -5), (4, 127, -1), (5, 3, -128), (20, 11, -4), (25, 60, -67), (32, 9, -9),
                                       (32, 100, -29)])
def test_matrix_profiles(pa, oracle, kw, group, dim, hi, lo):
    rng = np.random.default_rng(dim)
    alphabet = np.frombuffer(b"ABCDEFGHIJKLMNOPQRSTUVWXYZ012345"[:dim], np.uint8)
    scores = rng.integers(lo, 1, (dim, dim))
    scores[np.arange(dim), np.arange(dim)] = rng.integers(1, hi + 1, dim)
    scores[0, 0], scores[-1, 0] = hi, lo if dim > 1 else hi
    matrix = (bytes(alphabet), [int(x) for x in scores.ravel()])
    _run(pa, oracle, _batch(pa, dim, alphabet), group, kw, matrix=matrix)


@pytest.mark.parametrize("kw", MODES, ids=["global", "local", "free_column", "free_row"])
@pytest.mark.parametrize("group", [0, 4, 8, 16, 32])
@pytest.mark.parametrize("match,mismatch,alphabet,width", [(4, -5, b"ACGTN", 0), (3, 0, b"ACGT", 32), (300, -200, b"ACGT", 0),
                                                           (2, 1, b"ACGTacgt", 0), (2, -3, b"ACGT", 32)])
def test_bytes_and_tables(pa, oracle, kw, group, match, mismatch, alphabet, width):
    letters = np.frombuffer(alphabet, np.uint8)
    batch = _batch(pa, 50 + match, letters)
    if width == 0 and abs(match) < 128:                  # every sequence2 holds a byte outside A/C/G/T
        t, to = batch[2].copy(), batch[3].astype(np.int64)
        t[to[:-1]] = letters[-1]
        batch = (batch[0], batch[1], t, batch[3])
    _run(pa, oracle, batch, group, kw, match=match, mismatch=mismatch, width=width)
