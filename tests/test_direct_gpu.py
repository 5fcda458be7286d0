"""The unpartitioned join (one cooperative kernel) against the oracle and the partitioned join: step and
tile remainders, both build sides, long buckets, the limits of the rule that chooses it."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from gpu_helpers import assert_same_pairs, run_device

pytestmark = pytest.mark.gpu
MAX_BUILD = 3 << 20


def _join(bj, oracle, torch, data, launches=1, **cfg):
    exp = oracle.pairs(*data)
    n0 = bj.kernel_launches()
    st, r, s, k = run_device(bj, torch, *data, cap=max(len(exp[0]), 1), **cfg)
    if launches:
        assert bj.kernel_launches() - n0 == launches  # the path under test ran
    assert st.count == len(exp[0])
    assert_same_pairs(oracle, r, s, *exp)
    if k is not None:
        key = dict(zip(data[3].tolist(), data[2].tolist()))
        assert all(key[v] == q for v, q in zip(s.tolist(), k.tolist()))
    return st


@pytest.mark.parametrize("n_r,n_s", [(1, 1), (1, 4096), (127, 129), (3275, 3277), (4097, 65_537), (65_537, 4097),
                                     (200_003, 1_000_001), (1_000_001, 300_007)])
@pytest.mark.parametrize("cfg", [dict(), dict(use_bloom=1), dict(use_bloom=1, bloom_bits_per_key=14.0),
                                 dict(use_bloom=1, partition_mode=1)], ids=["plain", "k7", "k10", "modulo"])
def test_sizes(bj, oracle, torch_cuda, n_r, n_s, cfg):
    st = _join(bj, oracle, torch_cuda, bj.gen_host(n_r + n_s, n_r, n_s, 0.3), **cfg)
    if not cfg:
        assert st.s_survivors == n_s
    else:  # the same filter as the partitioned join's: the same survivors
        p = run_device(bj, torch_cuda, *bj.gen_host(n_r + n_s, n_r, n_s, 0.3), partition_size=st.partition_size,
                       second_partition_size=st.second_partition_size, **cfg)[0]
        assert (st.s_survivors, st.bloom_num_bits) == (p.s_survivors, p.bloom_num_bits)


@pytest.mark.parametrize("bloom", [0, 1])
@pytest.mark.parametrize("build", ["r", "s"])
@pytest.mark.parametrize("copies", [2, 9, 10, 254, 255, 256, 700, 20_000])
def test_repeated_build_keys(bj, oracle, torch_cuda, copies, build, bloom):
    """Buckets at the edges of the lock-step walk (8), the counted length (255) and the listed pieces (256)."""
    rng = np.random.default_rng(copies)
    hot = np.repeat(np.array([7, 0x80000000, 0xFFFFFFFF], np.uint32), [copies, max(copies // 2, 1), 3])
    small = rng.permutation(np.concatenate([hot, np.arange(100, 20_100, dtype=np.uint32)]))
    big = rng.permutation(np.concatenate([np.arange(10_000, 60_000, dtype=np.uint32),
                                          np.array([7, 7, 0x80000000, 0xFFFFFFFF, 5], np.uint32)]))
    rk, sk = (small, big) if build == "r" else (big, small)
    data = (rk, np.arange(len(rk), dtype=np.uint32), sk, np.arange(len(sk), dtype=np.uint32))
    _join(bj, oracle, torch_cuda, data, use_bloom=bloom, emit_key=True)


def test_one_key(bj, oracle, torch_cuda):
    """Every row of both sides has the same key: one bucket, and more pieces than the list holds."""
    rk, sk = np.full(5000, 0xDEADBEEF, np.uint32), np.full(700, 0xDEADBEEF, np.uint32)
    data = (rk, np.arange(5000, dtype=np.uint32), sk, np.arange(700, dtype=np.uint32))
    assert _join(bj, oracle, torch_cuda, data).count == 5000 * 700


@pytest.mark.parametrize("copies,rows,n_r,n_s,bloom", [
    (100_000, 200, 0, 500_000, 0), (100_000, 200, 0, 500_000, 1),  # few rows of long buckets: 400 pieces each
    (300, 60_000, 0, 140_000, 0),           # more rows than the list holds (32768), walked where they are met
    (5000, 3000, 0, 3000, 0),               # more rows than it holds of more entries than a warp may walk: rounds
    (2100, 34_000, 0, 140_000, 1),          # rounds behind the filter
    (2100, 34_000, 3_200_000, 20_000, 1),   # S's survivors build, rounds over R's rows
])
def test_hot_key_on_both_sides(bj, oracle, torch_cuda, copies, rows, n_r, n_s, bloom):
    """A key with many copies on the build side whose streamed rows lie side by side, as in a sorted relation.
    Exact pairs, and no slower than a small multiple of the partitioned join (a warp that walked its own
    rows' buckets while the others waited took over a hundred times as long)."""
    t = torch_cuda
    if n_r > n_s:
        copies, rows = rows, copies  # of the streamed R and of S
    rk = t.arange(2, 2 * max(n_r, copies) + 2, 2, dtype=t.int32, device="cuda")
    sk = t.arange(1, 2 * n_s + 1, 2, dtype=t.int32, device="cuda")
    rk[len(rk) // 3 if n_r > copies else 0:][:copies] = 0
    sk[n_s // 3 if n_s > rows else 0:][:rows] = 0
    r0, s0 = int((rk == 0).nonzero()[0]), int((sk == 0).nonzero()[0])
    rv, sv = (t.arange(len(k), dtype=t.int32, device="cuda") for k in (rk, sk))
    out = [t.empty(copies * rows, dtype=t.int32, device="cuda") for _ in range(2)]
    ms = []
    for cfg in (dict(), dict(table_capacity=4096)):
        with bj.Join(use_bloom=bloom, **cfg) as j:
            took = []
            for _ in range(4):
                e = [t.cuda.Event(enable_timing=True) for _ in range(2)]
                out[0].fill_(-1)
                n0 = bj.kernel_launches()
                e[0].record()
                j.run(rk, rv, len(rk), sk, sv, len(sk), out[0], out[1], copies * rows)
                e[1].record()
                assert (bj.kernel_launches() - n0 == 1) == (not cfg)
                assert j.stats().count == copies * rows
                took.append(e[0].elapsed_time(e[1]))
            pair = (out[0].long() - r0) * rows + (out[1] - s0)
            assert t.equal(pair.sort().values, t.arange(copies * rows, device="cuda"))
        ms.append(min(took[1:]))
    assert ms[0] < 4 * ms[1] + 1.0, ms


@pytest.mark.parametrize("n_r,n_s,direct", [(MAX_BUILD, 4_000_000, True), (MAX_BUILD + 1, 4_000_000, False),
                                            (5_000_000, MAX_BUILD, True)])
@pytest.mark.parametrize("bloom", [0, 1])
def test_limits(bj, oracle, torch_cuda, n_r, n_s, direct, bloom):
    n0 = bj.kernel_launches()
    _join(bj, oracle, torch_cuda, bj.gen_host(9, n_r, n_s, 0.2), launches=0, use_bloom=bloom)
    assert (bj.kernel_launches() - n0 == 1) == direct


M = 1 << 20


@pytest.mark.parametrize("n_r,n_s,many,bloom,direct", [
    (M, 24 * M, 1, 0, True), (M, 24 * M + 1, 1, 0, False), (M, 48 * M, 0, 0, True), (M, 48 * M + 1, 0, 0, False),
    (65_535, 24 * M + 1, 0, 1, False), (65_536, 24 * M + 1, 0, 1, True),  # a small filter
    (8191, 24 * M + 1, 0, 0, False), (8191, 24 * M, 0, 0, True),          # few rows
    (8191, 4 * M, 1, 1, True), (8191, 4 * M + 1, 1, 0, False), (8191, 4 * M + 1, 0, 1, False), (8192, 4 * M + 1, 1, 1, True),
    (48 * M, M, 1, 0, True), (48 * M, 8192, 1, 0, True), (24 * M + 1, 8191, 1, 0, False), (24 * M + 1, 8191, 0, 0, True)])
def test_limits_of_the_longer_side(bj, torch_cuda, n_r, n_s, many, bloom, direct):
    """Where the partitioned join is the faster one it is taken: many pairs asked for, a filter or a smaller
    side of few lines. Both give the same count."""
    t = torch_cuda
    d = [t.empty(n, dtype=t.int32, device="cuda") for n in (n_r, n_r, n_s, n_s)]
    bj.gen_device(6, n_r, n_s, 0.05, 0.0, *d)
    cap = max(n_r, n_s) // (4 if min(n_r, n_s) < 262_144 else 2) - (not many)
    out = [t.empty(cap, dtype=t.int32, device="cuda") for _ in range(2)]
    counts = []
    for cfg in (dict(), dict(table_capacity=4096)):
        with bj.Join(use_bloom=bloom, **cfg) as j:
            n0 = bj.kernel_launches()
            j.run(*d[:2], n_r, *d[2:], n_s, *out, cap)
            assert (bj.kernel_launches() - n0 == 1) == (direct and not cfg)
            counts.append(j.stats().count)
    assert counts[0] == counts[1] == int(0.05 * n_s)


@pytest.mark.parametrize("n_r,n_s,direct", [(3_000_000, 3_000_000, True),  # one copy after the other, then the join
                                            (7_500_000, 1 << 20, True), (7_500_000, (1 << 20) + 1, False),
                                            (2 << 20, 7_500_000, True), ((2 << 20) + 1, 7_500_000, False)])
def test_host_joins_overlap_the_copy_of_s(bj, oracle, n_r, n_s, direct):
    data = bj.gen_host(12, n_r, n_s, 0.1)
    exp = oracle.pairs(*data)
    with bj.Join(use_bloom=1) as j:
        n0 = bj.kernel_launches()
        cnt, r, s = j.run_host(*data, capacity=len(exp[0]))
        assert (bj.kernel_launches() - n0 == 1) == direct
    assert cnt == len(exp[0])
    assert_same_pairs(oracle, r, s, *exp)


@pytest.mark.parametrize("bloom", [0, 1])
@pytest.mark.parametrize("over", [("rv", "sv"), ("rk", "sk"), ("sv", "rv")])
def test_pairs_that_replace_the_inputs(bj, oracle, torch_cuda, over, bloom):
    """Outputs in the memory of inputs (here 10 words into them), as the partitioned join allows."""
    names = ("rk", "rv", "sk", "sv")
    data = bj.gen_host(15, 300_000, 400_000, 0.5)
    exp = oracle.pairs(*data)
    n = len(exp[0])
    d = {k: torch_cuda.from_numpy(a.view(np.int32)).cuda() for k, a in zip(names, data)}
    out = [d[k][10:10 + n] for k in over]
    with bj.Join(use_bloom=bloom) as j:
        j.run(d["rk"], d["rv"], 300_000, d["sk"], d["sv"], 400_000, *out, n)
        assert j.stats().count == n
    assert_same_pairs(oracle, *(o.cpu().numpy().view(np.uint32) for o in out), *exp)


SOME_SMS = """
import torch, brig_join as bj
t = torch.empty(1, device="cuda")
green = torch.cuda.GreenContext.create(16, 0)
green.set_context()
st = torch.cuda.Stream()
with torch.cuda.stream(st):
    for n, cfg in ((1_000_000, {}), (1_000_000, dict(use_bloom=1)), (1 << 24, dict(use_bloom=1, use_cuda_graph=1))):
        d = [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(4)]
        bj.gen_device(1, n, n, 0.1, 0.0, *d, stream=st.cuda_stream)
        out = [torch.empty(n // 8, dtype=torch.int32, device="cuda") for _ in range(2)]
        with bj.Join(**cfg) as j:
            for _ in range(2):
                j.run(*d[:2], n, *d[2:], n, *out, n // 8, stream=st.cuda_stream)
                print(j.stats().count)
green.pop_context()
"""


def test_stream_with_some_of_the_sms(torch_cuda):
    """A stream of a context that owns 16 SMs cannot hold the cooperative grid: the join runs all the same."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.path.join(root, "brig-join_b200"))
    r = subprocess.run([sys.executable, "-c", SOME_SMS], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split() == ["100000"] * 4 + ["1677721"] * 2


def test_misaligned_overflow_and_reuse(bj, oracle, torch_cuda):
    data = bj.gen_host(3, 70_001, 90_003, 0.4)
    exp = oracle.pairs(*data)
    with bj.Join(use_bloom=1) as j:
        for cap in (len(exp[0]), 1000, 0, len(exp[0])):
            st, r, s, _ = run_device(bj, torch_cuda, *data, cap=cap, handle=j, offset=(1, 2, 3, 1))
            assert st.count == len(exp[0]) and st.overflow == (cap < len(exp[0])) and len(r) == cap
            if cap == len(exp[0]):
                assert_same_pairs(oracle, r, s, *exp)
            else:
                assert set(zip(r.tolist(), s.tolist())) <= set(zip(exp[0].tolist(), exp[1].tolist()))


@pytest.mark.parametrize("path", [dict(), dict(table_capacity=4096)], ids=["default", "partitioned"])
def test_a_captured_run_is_refused(bj, oracle, torch_cuda, path):
    """Under a caller's stream capture no run is taken, and the handle runs again after it."""
    torch, cu = torch_cuda, ctypes.CDLL("libcuda.so.1")
    data = bj.gen_host(3, 5000, 9000, 0.4)
    exp = oracle.pairs(*data)
    d = [torch.from_numpy(x.view(np.int32)).cuda() for x in data]
    out = [torch.empty(len(exp[0]), dtype=torch.int32, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    with bj.Join(**path) as j:
        for _ in range(2):  # a handle's first run, and one after another
            stream, graph = torch.cuda.Stream(), ctypes.c_void_p()
            h = ctypes.c_void_p(stream.cuda_stream)
            assert cu.cuStreamBeginCapture_v2(h, 0) == 0  # CU_STREAM_CAPTURE_MODE_GLOBAL
            try:
                with pytest.raises(bj.BrigError):
                    j.run(d[0], d[1], 5000, d[2], d[3], 9000, *out, len(exp[0]), stream=stream.cuda_stream)
            finally:
                if cu.cuStreamEndCapture(h, ctypes.byref(graph)) == 0 and graph:
                    cu.cuGraphDestroy(graph)
            st, r, s, _ = run_device(bj, torch, *data, cap=len(exp[0]), handle=j)
            assert st.count == len(exp[0])
            assert_same_pairs(oracle, r, s, *exp)
