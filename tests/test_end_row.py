"""Free end of the last row in the short-pair kernel: maxima early and late in sequence1, ties (the
smallest end wins), values that fall below the 16-bit floor afterwards, two pairs of different
lengths in one unit, every strip remainder; against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = [1, 3, 4, 5, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 300]


@pytest.mark.parametrize("group", [4, 8, 16, 32])
@pytest.mark.parametrize("width,variant", [(0, 9), (0, 10), (32, -1)])
@pytest.mark.parametrize("scores", [(2, -4, -4, -2), (40, -30, -9, -1), (1, -1, -1, -1)])
@pytest.mark.parametrize("both", [False, True])
def test_last_row(built_lib, oracle, group, width, variant, scores, both):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pairwise_aligner_gb300 as pa
    rng = np.random.default_rng(group)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    s1, s2 = [], []
    for n in ROWS:
        read = acgt[rng.integers(0, 4, n)]
        for pad in (0, 7, 150, 900):
            left, right = acgt[rng.integers(0, 4, pad)], acgt[rng.integers(0, 4, 2 * pad)]
            # the read early, twice (a tie), late, not at all
            for parts in ([read, right], [left, read, left, read], [left, left, read], [right]):
                s1.append(b"".join(bytes(x) for x in parts))
                s2.append(bytes(read))
    batch = pa.pack(s1) + pa.pack(s2)
    match, mismatch, open_, ext = scores
    free = dict(first_column_free=True, first_row_free=False, last_column_free=True, last_row_free=both)
    conf = dict(local=False, match=match, mismatch=mismatch, gap_open=open_, gap_extension=ext, width_hint=width, **free)
    ctx = pa.Context(0, group_threads=group, kernel_variant=variant)
    res = pa.Aligner(conf, context=ctx).compute_arrays(*batch)
    ctx.close()
    want = oracle.align_batch(oracle.make_cfg(match, mismatch, open_, ext, local=False, **free), *batch)
    for got, exp in zip((res["score"], res["end1"], res["end2"]), want):
        assert np.array_equal(got, exp)
