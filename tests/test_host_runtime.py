"""The library's host logic on a make-believe CUDA runtime (cpp/host_runtime.cpp): two devices, no
kernel runs, every launch, allocation and occupancy query is on record."""
from __future__ import annotations

import ctypes
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

from conftest import REPO


class HostRuntime:
    def __init__(self, path):
        from pairwise_aligner_gb300 import _lib
        self.path = path
        self._lib = _lib
        self.lib = _lib.load(path)
        for name, res in (("events", ctypes.c_char_p), ("most", ctypes.c_size_t), ("reset", None), ("limit", None)):
            fn = getattr(self.lib, "host_runtime_" + name)
            fn.restype = res
            setattr(self, "_" + name, fn)
        self._limit.argtypes = [ctypes.c_size_t]

    def context(self, device=0, **opt):
        o = self._lib.PaOptions()
        o.kernel_variant = -1
        for k, v in opt.items():
            setattr(o, k, v)
        p = ctypes.c_void_p()
        assert self.lib.pa_create(ctypes.byref(p), device, ctypes.byref(o)) == 0
        return p

    def matrix(self, ctx, dim, top=9):
        symbols = np.arange(65, 65 + dim, dtype=np.uint8)
        scores = np.where(np.eye(dim), top, -3).astype(np.int32)
        return self.lib.pa_set_substitution_matrix(ctx, symbols.ctypes.data, dim, scores.ctypes.data)

    def align_device(self, ctx, n, b1, b2, local=True, matrix=False, match=1, mismatch=-4, free=False, width=0):
        """One device call; nothing reads the (made-up) buffers."""
        f = int(local or free)
        cfg = self._lib.PaConfig(int(local) | (self._lib.PA_SCORE_MATRIX if matrix else 0), match, mismatch, -6, -1,
                                 f, f, f, f, width, 0)
        at = [ctypes.c_void_p(0x10000 * k) for k in range(1, 6)]
        return self.lib.pa_align_batch_device(ctx, ctypes.byref(cfg), at[0], at[1], b1, at[2], at[3], b2, n, at[4], None,
                                              None)

    def events(self):
        text = self._events().decode()
        self._reset()
        return text.splitlines()


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    from pairwise_aligner_gb300 import build
    objs = build.objects()
    d = tmp_path_factory.mktemp("host_runtime")
    lib, group = str(d / "libpa_host.so"), d / "group.cu"
    group.write_text(f'#include "{build.CSRC}/pa_common.cuh"\n'
                     'extern "C" int dp_launch_group(const void *p) { return ((const pa::DpLaunch *)p)->G; }\n')
    nvcc = build.nvcc()
    subprocess.check_call([nvcc, *build.ARCH, "-std=c++17", "-Xcompiler", "-fPIC", "-diag-suppress", "177", "-shared",
                           "-cudart", "none", "-Xlinker", "-Bsymbolic", "-o", lib, str(group),
                           os.path.join(REPO, "tests", "cpp", "host_runtime.cpp"), *objs])
    return HostRuntime(lib)


def test_matrix_kernels_may_use_their_shared_memory_on_every_device(host):
    """The right to more than 48 KB of shared memory belongs to a device: a context on the second one
    needs its own, also when the first has asked for the same kernels already."""
    host.events()
    for device in (0, 1):
        ctx = host.context(device)
        for dim in (20, 32):                            # 40 and 64 KB of profiles
            assert host.matrix(ctx, dim) == 0
            for local, free in ((True, False), (False, False), (False, True)):
                assert host.align_device(ctx, 20000, 20000 * 300, 20000 * 300, local, True, free=free) == 0
        ev = host.events()
        assert not [e for e in ev if e.startswith("refused")], ev
        profile = [e for e in ev if "dp_short" in e and "Li2E" in e]
        assert profile and all(f"device {device}" in e for e in profile)
        host.lib.pa_destroy(ctx)


@pytest.mark.parametrize("local", [True, False])
def test_every_s32_variant_names_its_kernel(host, local):
    """pa_tuning::variant_s32 selects the inner loop of the s32 and byte-compare classes: 0..8 a form of
    the general kernel, whatever the default is; the default itself is the short-pair kernel."""
    mi, t = int(not local), host._lib.PaTuning()
    ctx = host.context(use_graphs=-1)
    assert host.lib.pa_get_tuning(ctx, ctypes.byref(t)) == 0
    for v in (None, 0, 4, 7, 9):
        if v is not None:
            t.variant_s32[mi] = v
            assert host.lib.pa_set_tuning(ctx, ctypes.byref(t)) == 0
        host.events()
        assert host.align_device(ctx, 5000, 5000 * 200, 5000 * 200, local) == 0
        s32 = [e for e in host.events() if re.search(r"dp_(short|kernel)I.*3L32", e)]
        assert len(s32) >= 2
        kind = "dp_kernel" if v is not None and v < 9 else "dp_short"
        assert all(kind in e for e in s32), (v, s32)
    host.lib.pa_destroy(ctx)


def test_group_size_of_the_general_kernel(host):
    """Its rule in global modes is its own: about eight units per resident warp (2,432 of them here), lane by
    lane; the short-pair kernel takes smaller groups for the same batches."""
    def groups(ctx, n, **kw):
        host.events()
        assert host.align_device(ctx, n, n * 288, n * 288, **kw) == 0
        got = {}
        for e in host.events():
            k = re.search(r"dp_(short|kernel)I.*(L16|L32)", e)
            if k:
                got.setdefault((k[1], k[2]), set()).add(int(e.split(" G ")[1]))
        return got
    general = host.context(use_graphs=-1, kernel_variant=4)
    assert groups(general, 60000, local=False, free=True) == {("kernel", "L16"): {32}, ("kernel", "L32"): {16}}
    matrix = host.context(use_graphs=-1)
    assert host.matrix(matrix, 20, top=400) == 0
    assert groups(matrix, 20000, matrix=True, local=False)[("kernel", "L32")] == {32}
    assert groups(matrix, 60000)[("short", "L16")] == {8}
    assert groups(general, 60000, local=True)[("kernel", "L16")] == {8}          # its best in local mode
    host.lib.pa_destroy(general)
    host.lib.pa_destroy(matrix)


def test_scratch_of_a_batch_without_room_for_long_pairs(host):
    """What a device call of short pairs may take: per byte of sequence1 and pair 28 bytes (score tables,
    boundary cells, slots), 16 per pair for the lists, the ring rows of 3.83 GB for long byte-compare
    pairs and the buckets of the sort.  Long pairs share the slots."""
    n, b = 1_000_000, 250_000_000
    for call in (dict(local=True), dict(local=False), dict(local=True, width=32)):
        host._reset()
        ctx = host.context()
        host._limit(28 * (b + n) + 16 * n + 3 * 304 * 8 * (65536 + 2) * 8 + 16 * 10**6 + 132 * b // 1024)
        assert host.align_device(ctx, n, b, b, **call) == 0
        host._limit(2**63)
        host.lib.pa_destroy(ctx)


def test_traceback_without_room_for_tagged_cells(host):
    """The tagged kernels need 16 bytes per column, the kernel with one warp per pair 8: a call that fits
    only with 8 runs on the latter."""
    n, m, k = 4000, 2500, 30
    s1, s2 = np.full(n * m, 65, np.uint8), np.full(n * k, 65, np.uint8)
    o1, o2 = np.arange(n + 1, dtype=np.uint64) * m, np.arange(n + 1, dtype=np.uint64) * k
    cfg = host._lib.PaConfig(0, 2, -3, -5, -1, 0, 0, 0, 0, 0, 0)
    out, aln, ops = np.zeros(n * 16, np.uint8), np.zeros(n * 16, np.uint8), np.zeros(n * (m + k), np.uint8)
    seen = []
    for cell in (16, 8):
        ctx = host.context()
        host.events()
        words = 4 * n * (m + 31) * 32                   # one pass of 256 rows
        host._limit(words + n * (m * 2 + k * 2 + 80) + cell * n * (m + 1) + 2 * 10**6)
        rc = host.lib.pa_traceback_batch(ctx, ctypes.byref(cfg), s1.ctypes.data, o1.ctypes.data, s2.ctypes.data,
                                         o2.ctypes.data, n, out.ctypes.data, aln.ctypes.data, ops.ctypes.data, None)
        host._limit(2**63)
        assert rc == 0, cell
        seen.append([re.search(r"k_t\w+", e)[0] for e in host.events() if "k_t" in e])
        host.lib.pa_destroy(ctx)
    assert all("k_tb" in x for x in seen[0]) and all("k_traceback" in x for x in seen[1]), seen


def test_no_occupancy_query_inside_a_capture(host, tmp_path):
    """What a launch needs to know of a kernel is asked when the context is made or the matrix set: the first
    calls of a process only enqueue while they are captured."""
    fresh = HostRuntime(shutil.copy(host.path, str(tmp_path / "fresh.so")))      # nothing asked yet
    ctx = fresh.context()
    assert fresh.matrix(ctx, 20) == 0
    for local, free in ((True, False), (False, False), (False, True)):
        for matrix in (False, True):
            for n, m in ((5000, 200), (300, 3000)):
                assert fresh.align_device(ctx, n, n * m, n * m, local, matrix, free=free) == 0
    assert not [e for e in fresh.events() if "in a capture" in e]
    fresh.lib.pa_destroy(ctx)


@pytest.mark.parametrize("band_mode", [0, 2])
def test_a_long_pair_without_room_for_ring_rows(host, band_mode):
    """Only long byte-compare pairs use the ring rows, 24 bytes per base of the longest sequence1 and resident
    warp (61 GB at 2^20): a call that has no room for them runs all the same."""
    m, n = 1 << 20, 2000
    s1, s2 = np.full(m, 65, np.uint8), np.full(n, 65, np.uint8)
    o1, o2 = np.array([0, m], np.uint64), np.array([0, n], np.uint64)
    cfg, out = host._lib.PaConfig(0, 2, -3, -5, -1, 0, 0, 0, 0, 0, band_mode), np.zeros(16, np.uint8)
    ctx = host.context()
    host.events()
    host._limit(2 * 10**9)
    rc = host.lib.pa_align_batch(ctx, ctypes.byref(cfg), s1.ctypes.data, o1.ctypes.data, s2.ctypes.data, o2.ctypes.data,
                                 1, out.ctypes.data, None)
    host._limit(2**63)
    assert rc == 0
    ev = host.events()
    assert band_mode or any("dp_longI" in e for e in ev)
    assert not any("dp_kernel_c" in e or "dp_kernel_team" in e for e in ev)
    host.lib.pa_destroy(ctx)
