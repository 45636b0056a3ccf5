"""Betweenness dependencies on the GPU (bfs_bc_run / bfs_bc_accumulate through
the C ABI) against the oracle's restatement of the reference's BC()
(apps/betweennessCentrality_simd/bc.cpp:1717-2097) and networkx's Brandes
values (tests/golden/bc_networkx.npz).

Path counts are unsigned integers and must be bit-exact.  Dependencies are
float sums whose order differs from the oracle's: |gpu - oracle| <=
1e-4 * (scale + 1), scale being the magnitude of the float sums behind each
value.  Repeated GPU runs must be bit-identical (fixed summation order).
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bc_case_names, bc_close, golden_case_names, load_bc_case, load_case

pytestmark = pytest.mark.gpu


def _check_source(oracle, arr, g, s):
    dep, sig, st = g.bc(int(s))
    osig, odep, ocost, oscale = oracle.bc_single(arr, int(s))
    np.testing.assert_array_equal(sig, osig, err_msg=f"path counts from {s}")
    ok = bc_close(dep, odep, oscale)
    bad = np.flatnonzero(~ok)
    assert ok.all(), f"source {s}: {bad[:6]} gpu {dep[bad[:6]]} oracle {odep[bad[:6]]}"
    assert st["status"] == 0
    reached = ocost >= 0
    assert st["reached"] == int(reached.sum())
    assert st["depth"] == int(ocost.max())
    assert st["edges_reached"] == int(arr["degrees"].astype(np.uint64)[reached].sum())
    assert (dep[~reached] == 0).all() and (sig[~reached] == 0).all()
    return dep, sig, st


@pytest.mark.parametrize("name", bc_case_names())
def test_bc_matches_oracle_and_networkx(native, oracle, name):
    import bfs_simd_benchmarks_gb300 as B
    c = load_bc_case(name)
    arr = oracle.arrays_from_edges(c["n"], c["src"], c["dst"], c["w"], c["s"])
    with B.Graph.from_edges(c["n"], c["src"], c["dst"], c["w"], c["s"]) as g:
        for i, s in enumerate(c["sources"]):
            dep, _, _ = _check_source(oracle, arr, g, s)
            _, _, cost, scale = oracle.bc_single(arr, int(s))
            want = c["delta"][i].copy()
            want[s] = float((cost >= 0).sum() - 1)
            ok = bc_close(dep, want, scale)
            assert ok.all(), f"{name} source {s} vs networkx: {np.flatnonzero(~ok)[:6]}"


@pytest.mark.parametrize("name", golden_case_names())
def test_bc_golden_graphs_deterministic(native, oracle, name):
    """Every golden graph (duplicate edges included), a repeat run bit-identical,
    and the byte-level gathers (bc_level_bytes = 1) giving the same bits as the
    8-byte ones (2)."""
    import bfs_simd_benchmarks_gb300 as B
    c = load_case(name)
    arr = oracle.arrays_from_edges(c["n"], c["src"], c["dst"], c["w"], c["s"])
    with B.Graph.from_edges(c["n"], c["src"], c["dst"], c["w"], c["s"]) as g:
        for s in c["sources"]:
            g.set_options(bc_level_bytes=2)
            dep, sig, _ = _check_source(oracle, arr, g, s)
            dep2, sig2, _ = g.bc(int(s))
            assert dep.tobytes() == dep2.tobytes() and sig.tobytes() == sig2.tobytes()
            g.set_options(bc_level_bytes=1)
            dep3, sig3, _ = g.bc(int(s))
            assert dep.tobytes() == dep3.tobytes() and sig.tobytes() == sig3.tobytes()


def test_bc_hubs_take_the_cta_path(native, oracle):
    """In- and out-degrees above 1024 (a whole CTA reduces those vertices)."""
    import bfs_simd_benchmarks_gb300 as B
    rng = np.random.default_rng(7)
    n = 6000
    src, dst = [], []
    # 0 -> 1..3000 -> 3001 (in-degree 3000) -> 3002..5999 (out-degree 2998)
    for v in range(1, 3001):
        src += [0, v]
        dst += [v, 3001]
    for v in range(3002, n):
        src.append(3001)
        dst.append(v)
    # random cross edges one level down keep path counts uneven
    extra_u = rng.integers(1, 3001, 4000)
    extra_v = rng.integers(3002, n, 4000)
    src = np.concatenate([np.array(src, np.uint32), extra_u.astype(np.uint32)])
    dst = np.concatenate([np.array(dst, np.uint32), extra_v.astype(np.uint32)])
    arr = oracle.arrays_from_edges(n, src, dst, 256, 4)
    with B.Graph.from_edges(n, src, dst, 256, 4) as g:
        for s in (0, 17, 3001):
            _check_source(oracle, arr, g, s)


def test_bc_many_big_vertices_in_one_level(native, oracle):
    """A level with more than 4096 big vertices (one CTA each) followed by a
    level of 1800 big vertices (chunked over the grid)."""
    import bfs_simd_benchmarks_gb300 as B
    rng = np.random.default_rng(11)
    first, pool = 4200, 1800
    n = 1 + first + pool
    src = [np.zeros(first, np.uint32)]
    dst = [np.arange(1, first + 1, dtype=np.uint32)]
    for v in range(1, first + 1):
        t = rng.choice(pool, 1100, replace=False).astype(np.uint32) + first + 1
        src.append(np.full(1100, v, np.uint32))
        dst.append(t)
    src = np.concatenate(src)
    dst = np.concatenate(dst)
    arr = oracle.arrays_from_edges(n, src, dst, 512, 8)
    with B.Graph.from_edges(n, src, dst, 512, 8) as g:
        for mode in (1, 2):
            g.set_options(bc_level_bytes=mode)
            _, _, st = _check_source(oracle, arr, g, 0)
            assert st["level_big"][1] == first and st["level_big"][2] == pool


def test_bc_deep_chain(native, oracle):
    """5000 levels: the level sort's keys far beyond one per warp range."""
    import bfs_simd_benchmarks_gb300 as B
    n = 5000
    src = np.arange(n - 1, dtype=np.uint32)
    dst = src + 1
    # a few shortcuts that create two shortest paths around some vertices
    src = np.concatenate([src, np.array([10, 100, 2000], np.uint32)])
    dst = np.concatenate([dst, np.array([12, 102, 2002], np.uint32)])
    arr = oracle.arrays_from_edges(n, src, dst, 64, 4)
    with B.Graph.from_edges(n, src, dst, 64, 4) as g:
        g.set_options(bc_level_bytes=1)   # deeper than 254 levels: the 8-byte gathers are used anyway
        _check_source(oracle, arr, g, 0)
        _check_source(oracle, arr, g, 1500)


def test_bc_rmat18_permuted(native, oracle):
    import bfs_simd_benchmarks_gb300 as B
    n, m = 1 << 18, 1 << 22
    src, dst = B.gen_rmat(n, m, 0.57, 0.19, 0.19, seed=181, dedup=True, no_self_loops=True, permute=True)
    arr = oracle.arrays_from_edges(n, src, dst, 1024, 16)
    deg = arr["degrees"]
    with B.Graph.from_edges(n, src, dst, 1024, 16) as g:
        for mode in (1, 2):
            g.set_options(bc_level_bytes=mode)
            for s in np.flatnonzero(deg > 0)[[3, 999]]:
                _check_source(oracle, arr, g, int(s))


def test_bc_accumulate_matches_networkx_and_oracle(native, oracle):
    import bfs_simd_benchmarks_gb300 as B
    c = load_bc_case("rmat10_w64_s3")
    n = c["n"]
    arr = oracle.arrays_from_edges(n, c["src"], c["dst"], c["w"], c["s"])
    scale = np.zeros(n)
    for s in range(n):
        _, _, _, sc = oracle.bc_single(arr, s)
        sc = sc.copy()
        sc[s] = 0
        scale += sc
    with B.Graph.from_edges(n, c["src"], c["dst"], c["w"], c["s"]) as g:
        bc, st = g.betweenness(np.arange(n))
        assert st["num_sources"] == n and st["status"] == 0
        ok = bc_close(bc, c["bc"], scale)
        assert ok.all(), np.flatnonzero(~ok)[:8]
        # a subset of sources against the oracle's sum
        subset = np.array([5, 77, 300, 1023], np.uint32)
        part, _ = g.betweenness(subset)
        want = np.zeros(n)
        sc_sum = np.zeros(n)
        for s in subset:
            _, d, _, sc = oracle.bc_single(arr, int(s))
            d = d.astype(np.float64)
            d[s] = 0
            sc = sc.copy()
            sc[s] = 0
            want += d
            sc_sum += sc
        assert bc_close(part, want, sc_sum).all()


def test_bc_device_entry_points_match_host(native):
    import torch
    import bfs_simd_benchmarks_gb300 as B
    c = load_case("rmat12p_w100_s5")
    n = c["n"]
    with B.Graph.from_edges(n, c["src"], c["dst"], c["w"], c["s"]) as g:
        s = int(c["sources"][1])
        dep, sig, _ = g.bc(s)
        d_dep = torch.empty(n, dtype=torch.float32, device="cuda")
        d_sig = torch.empty(n, dtype=torch.int32, device="cuda")
        stream = torch.cuda.current_stream().cuda_stream
        g.bc_device(s, d_dep.data_ptr(), d_sig.data_ptr(), stream)
        torch.cuda.synchronize()
        assert g.bc_stats()["status"] == 0
        assert d_dep.cpu().numpy().tobytes() == dep.tobytes()
        assert d_sig.cpu().numpy().view(np.uint32).tobytes() == sig.tobytes()
        srcs = c["sources"]
        g.set_options(bc_batch=0)   # the device accumulation runs one source at a time
        host_bc, _ = g.betweenness(srcs)
        acc = torch.zeros(n, dtype=torch.float32, device="cuda")
        g.betweenness_device(srcs, acc.data_ptr(), stream)
        g.betweenness_device(srcs, acc.data_ptr(), stream)   # adds: twice the sum
        torch.cuda.synchronize()
        np.testing.assert_allclose(acc.cpu().numpy(), 2 * host_bc, rtol=1e-6, atol=1e-6)


def test_bc_arguments(native):
    import bfs_simd_benchmarks_gb300 as B
    from bfs_simd_benchmarks_gb300 import _native as N
    c = load_case("sparse15_w16_s2")
    with B.Graph.from_edges(c["n"], c["src"], c["dst"], c["w"], c["s"]) as g:
        with pytest.raises(N.BfsError) as e:
            g.bc(c["n"])
        assert e.value.status == N.BFS_EARG
        with pytest.raises(N.BfsError):
            g.betweenness(np.array([0, c["n"] + 5], np.uint32))
        # a source with no out-edges reaches nothing else
        deg = np.bincount(c["src"], minlength=c["n"])
        s = int(np.flatnonzero(deg == 0)[0])
        dep, sig, st = g.bc(s)
        assert st["reached"] == 1 and sig[s] == 1 and (dep == 0).all()


def _sink_graph(k, tail, others=0):
    """0 -> k vertices -> one sink without out-edges, 3 of them also -> a path of
    `tail` more levels; `others` more in-edges of the sink come from the path's end
    (with them, the sink's level has far more in-edges than the level before has
    out-edges).  The sink's level is not the deepest."""
    mids = np.arange(1, k + 1)
    sink, path = k + 1, np.arange(k + 2, k + 2 + tail)
    far = np.arange(path[-1] + 1, path[-1] + 1 + others)
    src = [np.zeros(k, int), mids, mids[:3], path[:-1], np.full(others, path[-1]), far]
    dst = [mids, np.full(k, sink), np.full(3, path[0]), path[1:], far, np.full(others, sink)]
    return int(path[-1]) + 1 + others, np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32)


@pytest.mark.parametrize("k, tail, others", [(1024, 2, 0), (1025, 1, 0), (1025, 3, 0), (5000, 2, 0), (3, 2, 1100), (40, 3, 5000)])
def test_bc_hub_without_out_edges(native, oracle, k, tail, others):
    """Sinks with many in-edges on a level that others follow, reached by a pulled
    or a pushed level: through every entry point that takes one source at a time."""
    import torch
    import bfs_simd_benchmarks_gb300 as B
    n, src, dst = _sink_graph(k, tail, others)
    arr = oracle.arrays_from_edges(n, src, dst, 256, 4)
    with B.Graph.from_edges(n, src, dst, 256, 4) as g:
        g.set_options(bc_batch=0)
        for mode in (1, 2):
            g.set_options(bc_level_bytes=mode)
            for s in (0, 1):
                dep, _, _ = _check_source(oracle, arr, g, s)
                total, _ = g.betweenness(np.array([s], np.uint32))
                want = dep.copy()
                want[s] = 0
                np.testing.assert_array_equal(total, want)
                acc = torch.zeros(n, dtype=torch.float32, device="cuda")
                g.betweenness_device(np.array([s], np.uint32), acc.data_ptr(), torch.cuda.current_stream().cuda_stream)
                torch.cuda.synchronize()
                np.testing.assert_array_equal(acc.cpu().numpy(), want)


@pytest.mark.parametrize("width, height, both", [(200, 200, False), (150, 170, True), (60, 300, True)])
def test_bc_sums_past_the_largest_float(native, oracle, width, height, both):
    """Street grids: path counts wrap, and sums of their reciprocals become infinite, of
    either sign, or NaN where both meet: at the same vertices as in the oracle."""
    import bfs_simd_benchmarks_gb300 as B
    y, x = np.divmod(np.arange(width * height), width)
    src, dst = [], []
    for dy, dx in ((0, 1), (1, 0)) + (((0, -1), (-1, 0)) if both else ()):
        ok = (y + dy >= 0) & (y + dy < height) & (x + dx >= 0) & (x + dx < width)
        src.append((y * width + x)[ok])
        dst.append(((y + dy) * width + x + dx)[ok])
    src, dst = np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32)
    n = width * height
    arr = oracle.arrays_from_edges(n, src, dst, 256, 4)
    osig, odep, _, _ = oracle.bc_single(arr, 0)
    assert np.isposinf(odep).any() and np.isneginf(odep).any() and np.isnan(odep).any()
    with B.Graph.from_edges(n, src, dst, 256, 4) as g:
        for mode in (1, 2):
            g.set_options(bc_level_bytes=mode)
            dep, sig, _ = g.bc(0)
            np.testing.assert_array_equal(sig, osig)
            for kind in (np.isposinf, np.isneginf, np.isnan):
                np.testing.assert_array_equal(kind(dep), kind(odep))


def _layers(sizes, seed, per=3, back=0, hubs=()):
    """Layer i + 1's vertices get `per` edges each from random vertices of layer i (every
    one of them is reached); `back` edges from each later layer to the one before;
    hubs: (layer, extra in-edges from that layer's successors and from vertices that
    nothing reaches)."""
    rng = np.random.default_rng(seed)
    at = np.concatenate([[0], np.cumsum(sizes)])
    n = int(at[-1])
    src, dst = [], []
    for i in range(len(sizes) - 1):
        a, b = np.arange(at[i], at[i + 1]), np.arange(at[i + 1], at[i + 2])
        src.append(rng.choice(a, per * b.size))
        dst.append(np.repeat(b, per))
        if back:
            src.append(rng.choice(b, back * b.size))
            dst.append(rng.choice(a, back * b.size))
    for layer, extra in hubs:
        island = np.arange(n, n + extra)
        src.append(island)
        dst.append(np.full(extra, at[layer]))
        n += extra
    return n, np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32)


def _degrees(out, inn, seed):
    """0 -> hubs -> pool -> hubs' -> end: hubs with the given out-degrees, hubs' with the given in-degrees."""
    rng = np.random.default_rng(seed)
    pool = max(max(out), max(inn)) + 50
    h, p = np.arange(1, 1 + len(out)), np.arange(1 + len(out), 1 + len(out) + pool)
    k = np.arange(p[-1] + 1, p[-1] + 1 + len(inn))
    src, dst = [np.zeros(len(out), int)], [h]
    for v, d in zip(h, out):
        src.append(np.full(d, v))
        dst.append(rng.choice(p, d, replace=False))
    src.append(np.full(pool, h[0]))  # the whole pool is on one level
    dst.append(p)
    for v, d in zip(k, inn):
        src.append(rng.choice(p, d, replace=False))
        dst.append(np.full(d, v))
    src.append(k)
    dst.append(np.full(len(inn), k[-1] + 1))
    return int(k[-1]) + 2, np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32)


BC_CASES = {
    # chunks of 512 edges of vertices with more than 1024, half-warps and lanes below
    "chunks": _degrees([1023, 1024, 1025, 1535, 1536, 1537, 2048, 2049], [1024, 1025, 1536, 1537, 2049, 4000], 1),
    "bands": _degrees([7, 8, 9, 31, 32, 33, 63, 64, 65, 512, 513], [1, 7, 8, 9, 15, 16, 17, 32, 33, 128, 129], 2),
    # sort counters in shared memory up to 32 levels; traced levels (and pushing) up to 64
    **{f"levels_{k}": _layers([1] + [5 + i % 7 for i in range(k - 1)], k, back=1) for k in (31, 32, 33, 63, 64, 65, 66)},
    # levels reached by few of their in-edges are pushed: one, two in a row, the last one, pulled ones around them
    "push_first": _layers([1, 3, 400, 400, 50], 3, hubs=[(1, 700), (2, 5000)]),
    "push_two": _layers([1, 40, 60, 900, 30], 4, back=1, hubs=[(2, 3000), (3, 9000)]),
    "push_last": _layers([1, 200, 600, 20], 5, hubs=[(3, 6000)]),
    "push_every": _layers([1, 4, 9, 30, 20], 6, hubs=[(i, 2000) for i in range(1, 5)]),
    "push_none": _layers([1, 500, 500, 500], 7, per=8),
    "push_deep": _layers([1] + [6] * 70, 8, hubs=[(i, 300) for i in (10, 62, 63, 64, 65, 70)]),
}
# lists that start at every edge number modulo 4 and end at the array's last edges
for _k in range(4):
    _n, _s, _d = _layers([1, 9, 40, 30, 6], 20 + _k, per=5, back=2)
    BC_CASES[f"edges_mod_{(_s.size - _k) % 4}"] = (_n, _s[:_s.size - _k], _d[:_s.size - _k])


@pytest.mark.parametrize("name", list(BC_CASES))
def test_bc_shapes(native, oracle, name):
    """The edges of k_bc's rules, in both gather modes, on graphs built on the host and on the device."""
    import bfs_simd_benchmarks_gb300 as B
    n, src, dst = BC_CASES[name]
    arr = oracle.arrays_from_edges(n, src, dst, 256, 4)
    for device_build in (False, True):
        with B.Graph.from_edges(n, src, dst, 256, 4, device_build=device_build) as g:
            g.set_options(bc_batch=0)
            for mode in (1, 2):
                g.set_options(bc_level_bytes=mode)
                for s in (0, 2, n // 2):
                    dep, _, _ = _check_source(oracle, arr, g, s)
                    total, st = g.betweenness(np.array([s], np.uint32))
                    dep[s] = 0
                    np.testing.assert_array_equal(total, dep)
