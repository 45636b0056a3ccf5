"""Single-source traversals whose frontiers are small enough for one CTA to take
several steps by itself: the edges of that rule (2048 vertices and out-edges,
128 steps, 2^18 vertices) and what it hands back to the whole grid, against the
oracle (levels and direction trace bit-exact, parents a valid tree)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _star(leaves, fan):
    """0 -> leaves 1..d; leaf i -> fan[i % len(fan)] of its own grandchildren and one shared vertex."""
    src, dst, n = [0] * leaves, list(range(1, leaves + 1)), leaves + 2
    shared = leaves + 1
    for i in range(leaves):
        for _ in range(fan[i % len(fan)]):
            src.append(i + 1)
            dst.append(n)
            n += 1
        src.append(i + 1)
        dst.append(shared)
    return n, src, dst


def _chain(levels, width, n=0):
    """`levels` layers of `width` vertices, each layer's vertices to all of the next; isolated vertices up to n."""
    src, dst = [], []
    for l in range(levels):
        for i in range(width):
            for j in range(width):
                src.append(l * width + i)
                dst.append((l + 1) * width + j)
    return max(n, (levels + 1) * width), src, dst


def _ladder_into_hub(hub):
    """A chain of 5, a hub of `hub` out-edges, and a second chain behind its last leaf."""
    n, src, dst = 5, [0, 1, 2, 3], [1, 2, 3, 4]
    first = n
    src += [4] * hub
    dst += range(first, first + hub)
    n += hub
    for i in range(6):
        src.append(n - 1)
        dst.append(n)
        n += 1
    return n, src, dst


CASES = {
    "star_2047": _star(2047, [0]),
    "star_2048": _star(2048, [0]),
    "star_2049": _star(2049, [0]),
    "star_grows": _star(300, [1, 9, 0, 40]),
    "star_edges_past_cap": _star(200, [10]),
    "chain_127": _chain(127, 1),
    "chain_128": _chain(128, 1),
    "chain_129": _chain(129, 1),
    "chain_300x3": _chain(300, 3),
    "layers_45": _chain(6, 45),
    "layers_46": _chain(6, 46),
    "chain_2p18": _chain(140, 2, 1 << 18),
    "chain_2p18_plus": _chain(140, 2, (1 << 18) + 1),
    "hub_2048": _ladder_into_hub(2048),
    "hub_5000": _ladder_into_hub(5000),
}


@pytest.mark.parametrize("rule", [0, 1])
@pytest.mark.parametrize("degree_order", [False, True])
@pytest.mark.parametrize("name", list(CASES))
def test_small_frontiers(native, oracle, name, degree_order, rule):
    import bfs_simd_benchmarks_gb300 as B
    n, src, dst = CASES[name]
    src, dst = np.asarray(src + src[:3], np.uint32), np.asarray(dst + dst[:3], np.uint32)  # with duplicate edges
    arr = oracle.arrays_from_edges(n, src, dst, 64, 4)
    deg = arr["degrees"].astype(np.uint64)
    with B.Graph.from_edges(n, src, dst, 64, 4, degree_order=degree_order) as g:
        g.set_options(switch_rule=rule)
        for s in (0, 1):
            ref = oracle.bfs_levels(arr, s)
            lev, par, st = g.run(s)
            np.testing.assert_array_equal(lev, ref)
            assert oracle.check_parents(arr, s, lev, par) == 0
            assert st["status"] == 0
            assert st["num_steps"] == ref.max() + 1
            assert st["reached"] == int((ref >= 0).sum())
            assert st["edges_traversed"] == int(deg[ref >= 0].sum())
            if rule == 0:
                _, _, trace, _ = oracle.bfs_hybrid(arr, s)
                k = min(len(trace), st["num_steps"], 256)
                assert list(st["trace"][:k]) == list(trace[:k])


def test_a_smaller_graph_leaves_a_larger_one_callable(native, oracle):
    """Each graph's traversals ask for their own amount of shared memory, whatever was built since."""
    import bfs_simd_benchmarks_gb300 as B
    n = 1 << 15
    src, dst = B.gen_rmat(n, 4 * n, seed=77, permute=True)
    arr = oracle.arrays_from_edges(n, src, dst, 1024, 16)
    s = int(B.pick_sources(arr["degrees"], 1, seed=3)[0])
    ref = oracle.bfs_levels(arr, s)
    with B.Graph.from_edges(n, src, dst, 1024, 16) as g:
        with B.Graph.from_edges(3, [0, 1], [1, 2], 64, 4) as small:
            for bottom_up in ("pull", "stream"):
                for mode in ("persistent", "stepwise"):
                    g.set_options(bottom_up=bottom_up, mode=mode)
                    lev, _, st = g.run(s)
                    assert st["status"] == 0
                    np.testing.assert_array_equal(lev, ref)
            np.testing.assert_array_equal(small.run(0)[0], [0, 1, 2])


def _mixed(n, seed):
    """Random edges, a hub whose long in-edge list starts at unreachable vertices, a hub with many out-edges."""
    rng = np.random.default_rng(seed)
    src = [rng.integers(0, n, size=3 * n)]
    dst = [rng.integers(0, n, size=3 * n)]
    if n > 1000:
        island = np.arange(n - n // 8, n)          # only out-edges: never reached
        keep = dst[0] < n - n // 8
        src[0], dst[0] = src[0][keep], dst[0][keep]
        src.append(np.repeat(island, 2)[:9000])
        dst.append(np.full(src[-1].size, 5))
        src.append(np.full(3000, 7))
        dst.append(rng.integers(0, n // 2, size=3000))
    return np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32)


@pytest.mark.parametrize("n", [1, 31, 33, 1024, 1025, 4097, 20_000, 65_536, 65_537, 98_304, 98_305])
def test_one_cluster_traversal(native, oracle, n):
    """Small graphs are traversed in one cluster: its sizes, both directions at every
    step and mixed ones, against the oracle and the whole grid's step sequence."""
    import bfs_simd_benchmarks_gb300 as B
    src, dst = _mixed(n, n)
    arr = oracle.arrays_from_edges(n, src, dst, 256, 4)
    deg = arr["degrees"].astype(np.uint64)
    with B.Graph.from_edges(n, src, dst, 256, 4) as g:
        for s in sorted({0, n // 3, min(7, n - 1)}):
            ref = oracle.bfs_levels(arr, s)
            for opts in ({}, {"switch_rule": 1}, {"to_dense_ratio": 1, "to_sparse_ratio": 1},
                         {"to_dense_ratio": 1 << 30, "to_sparse_ratio": 1 << 30}):
                g.set_options(**{"switch_rule": 0, "to_dense_ratio": 20, "to_sparse_ratio": 20, "ctas_per_sm": 0, **opts})
                lev, par, st = g.run(s)
                np.testing.assert_array_equal(lev, ref)
                assert oracle.check_parents(arr, s, lev, par) == 0
                assert st["reached"] == int((ref >= 0).sum()) and st["num_steps"] == ref.max() + 1
                assert st["edges_traversed"] == int(deg[ref >= 0].sum())
                assert (st["grid_ctas"] <= 16) == (n <= 65_536 or (n <= 98_304 and len(src) <= 4 * n))
                np.testing.assert_array_equal(g.run(s, parents=False)[0], ref)
                g.set_options(ctas_per_sm=2)
                lev2, _, st2 = g.run(s)
                assert st2["grid_ctas"] > 16
                np.testing.assert_array_equal(lev2, ref)
                for k in ("trace", "dense_steps", "td_edges", "td_vertices", "num_steps"):
                    assert st[k] == st2[k], (k, opts)


@pytest.mark.parametrize("ctas_per_sm", [0, 1])
@pytest.mark.parametrize("layers", ["few", "many"])
def test_grid_pull_lists(native, oracle, layers, ctas_per_sm):
    """The whole grid's bottom-up step on in-edge lists whose frontier source comes
    first, in the lane's share, in the queue's rounds, in the warp's rounds and
    never; top-down steps with and without the visited screen."""
    import bfs_simd_benchmarks_gb300 as B
    n = 200_003
    rng = np.random.default_rng(3)
    island = np.arange(n - 20_000, n)  # no in-edges: never reached
    src, dst = [rng.integers(0, 1000, size=4000)], [rng.integers(0, 1000, size=4000)]
    at = 1000
    for length in (1, 2, 3, 4, 5, 11, 12, 67, 68, 69, 131, 132, 133, 700):
        for _ in range(40):
            u = rng.choice(island, size=length)
            if rng.random() < 0.8:
                u[rng.integers(0, length)] = rng.integers(0, 1000)
            src.append(u)
            dst.append(np.full(length, at))
            at += 1
    last = np.arange(at, n - 20_000)
    per = 5 if layers == "many" else 1
    src.append(rng.integers(0, at, size=per * last.size))
    dst.append(np.repeat(last, per))
    if layers == "many":  # edges back to visited vertices, for the screened top-down steps
        src.append(np.repeat(last, 2))
        dst.append(rng.integers(0, n - 20_000, size=2 * last.size))
    src, dst = np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32)
    arr = oracle.arrays_from_edges(n, src, dst, 256, 4)
    with B.Graph.from_edges(n, src, dst, 256, 4, device_build=False) as g:
        for opts in ({}, {"switch_rule": 1}, {"to_dense_ratio": 1 << 30, "to_sparse_ratio": 1 << 30},
                     {"to_dense_ratio": 1 << 30, "to_sparse_ratio": 2}, {"to_dense_ratio": 1, "to_sparse_ratio": 1}):
            g.set_options(**{"switch_rule": 0, "to_dense_ratio": 20, "to_sparse_ratio": 20, "ctas_per_sm": ctas_per_sm, **opts})
            for s in (0, 17):
                lev, par, st = g.run(s)
                np.testing.assert_array_equal(lev, oracle.bfs_levels(arr, s))
                assert oracle.check_parents(arr, s, lev, par) == 0
                assert st["grid_ctas"] > 16


def test_grid_pull_queue_overflow(native, oracle):
    """More long in-edge lists in a work item than its queue holds."""
    import torch
    import bfs_simd_benchmarks_gb300 as B
    n = 4_200_000
    gen = torch.Generator(device="cuda")
    gen.manual_seed(9)
    island = 1000  # vertices n - 1000 ..: no in-edges
    heads = torch.arange(2, n - island, device="cuda", dtype=torch.int32).repeat_interleave(5)
    tails = torch.randint(n - island, n, (heads.numel(),), device="cuda", dtype=torch.int32, generator=gen)
    chain = torch.tensor([0, 1, 2, 3], device="cuda", dtype=torch.int32)
    src = torch.cat([tails, chain[:3]]).contiguous()
    dst = torch.cat([heads, chain[1:]]).contiguous()
    arr = oracle.csr_arrays(n, src.cpu().numpy().astype(np.uint32), dst.cpu().numpy().astype(np.uint32))
    with B.Graph.from_device_edges(n, src.data_ptr(), dst.data_ptr(), src.numel(), 1024, 16) as g:
        g.set_options(to_dense_ratio=1 << 30, to_sparse_ratio=1 << 30)
        for s in (0, n - 5):
            lev, par, st = g.run(s)
            np.testing.assert_array_equal(lev, oracle.bfs_levels(arr, s))
            assert oracle.check_parents(arr, s, lev, par) == 0
            assert st["dense_steps"] > 0


@pytest.mark.parametrize("wait_limit_us", [50, 200, 400])
def test_rounds_of_one_cta_fit_the_wait_limit(native, oracle, wait_limit_us):
    """300 top-down steps that one CTA takes (1,600 edges, some 8 us each) on a graph
    of more than 2^18 vertices: the wait of the other CTAs, of up to 128 of them,
    is not what runs out."""
    import bfs_simd_benchmarks_gb300 as B
    n, src, dst = _chain(300, 40, 300_000)
    src, dst = np.asarray(src, np.uint32), np.asarray(dst, np.uint32)
    with B.Graph.from_edges(n, src, dst, 1024, 16) as g:
        g.set_options(to_dense_ratio=1, wait_limit_us=wait_limit_us)
        arr = oracle.csr_arrays(n, src, dst)
        for s in (0, 41):
            lev, par, st = g.run(s)
            assert st["status"] == 0 and st["dense_steps"] == 0 and st["grid_ctas"] > 16
            np.testing.assert_array_equal(lev, oracle.bfs_levels(arr, s))
            assert oracle.check_parents(arr, s, lev, par) == 0


@pytest.mark.parametrize("n, used", [
    (1 << 22, np.arange(1 << 14)),                      # the first ids
    ((1 << 20) - 256, np.arange(3000)),                 # no list of blocks yet
    (1 << 20, np.arange(3000)),                         # the smallest graph with one
    ((1 << 20) + 77, np.arange((1 << 20) - 20_000, (1 << 20) + 77)),  # the last ones, the last block cut off
    (1_200_000, np.arange(200_001, 220_000)),
    (1_200_000, np.arange(0, 1_200_000, 300)),              # one in a block or none
    (1_200_000, np.arange(0, 1_200_000, 256)),              # one in every block
    (1_200_000, np.concatenate([np.arange(600_000), np.arange(800_000, 1_101_000)])),  # about three quarters of the blocks
    (100_000, np.array([99_999, 5])),
])
def test_grid_pull_of_sparse_ids(native, oracle, tmp_path, n, used):
    """Graphs whose edges are among some of the ids: the grid's bottom-up steps go through
    the blocks of the bitmap that have in-edges, and share them out."""
    import bfs_simd_benchmarks_gb300 as B
    rng = np.random.default_rng(n + used.size)
    src, dst = rng.choice(used, 12 * used.size).astype(np.uint32), rng.choice(used, 12 * used.size).astype(np.uint32)
    arr = oracle.csr_arrays(n, src, dst)
    path = str(tmp_path / "g.bin")
    s = int(src[0])
    ref = oracle.bfs_levels(arr, s)
    for how in ("host", "device", "degree order", "file"):
        if how == "file":
            g = B.Graph.load_binary(path)
        else:
            g = B.Graph.from_edges(n, src, dst, 1024, 16, device_build=how != "host", degree_order=how == "degree order")
            if how == "host":
                g.save(path)
        with g:
            for opts in ({}, {"to_dense_ratio": 1 << 30, "to_sparse_ratio": 1 << 30}, {"ctas_per_sm": 1},
                         {"mode": "stepwise"}):
                g.set_options(**{"to_dense_ratio": 20, "to_sparse_ratio": 20, "ctas_per_sm": 2, "mode": "persistent", **opts})
                lev, par, st = g.run(s)
                np.testing.assert_array_equal(lev, ref)
                assert oracle.check_parents(arr, s, lev, par) == 0
                assert st["reached"] == int((ref >= 0).sum())
                if "to_dense_ratio" in opts and used.size == 1 << 14:
                    # 512 words with in-edges, by 16 CTAs or more as long as most are unvisited
                    assert st["bu_groups"] >= 16


def test_grid_pull_without_in_edges(native):
    """No edges at all, and every step bottom-up: no block to go through."""
    import bfs_simd_benchmarks_gb300 as B
    none = np.zeros(0, np.uint32)
    with B.Graph.from_edges(70_000, none, none, 1024, 16) as g:
        g.set_options(ctas_per_sm=1, to_dense_ratio=1 << 30, to_sparse_ratio=1 << 30)
        lev, _, st = g.run(69_999)
        assert st["status"] == 0 and st["reached"] == 1 and lev[69_999] == 0 and (lev[:-1] == -1).all()


@pytest.mark.parametrize("where", ["cluster", "one CTA", "grid"])
def test_step_statistics(native, where):
    """Every step has its time and the first and last CTA's, the bottom-up steps their
    items, in each form of the traversal; a batch that runs as single traversals names
    their CTAs."""
    import torch
    import bfs_simd_benchmarks_gb300 as B
    n = 1 << (14 if where == "cluster" else 18)
    src, dst = B.gen_rmat(n, 16 * n, seed=9, permute=True)
    if where == "one CTA":
        n, src, dst = _chain(200, 3, 1 << 17)
        src, dst = np.asarray(src, np.uint32), np.asarray(dst, np.uint32)
    s = int(src[0])
    with B.Graph.from_edges(n, src, dst, 256, 4) as g:
        if where == "one CTA":
            g.set_options(to_dense_ratio=1)
        _, _, st = g.run(s)
        k = min(st["num_steps"], 256)
        step, lo, hi = (np.array(st[x][:k]) for x in ("step_ms", "step_work_min_ms", "step_work_max_ms"))
        assert (step > 0).all() and (lo > 0).all() and (lo <= hi).all() and (hi <= step).all()
        if where == "one CTA":
            assert (lo == step).sum() > k // 2
            return
        assert (st["grid_ctas"] <= 16) == (where == "cluster")
        assert st["dense_steps"] > 0 and st["bu_groups"] >= st["dense_steps"]
        g.set_options(batch_single_max=4)
        out = torch.empty((2, n), dtype=torch.uint8, device="cuda")
        b = g.run_batch_device(np.array([s, s], np.uint32), out.data_ptr(), torch.cuda.current_stream().cuda_stream, stats=True)
        assert b["single_source_runs"] == 2 and b["grid_ctas"] == st["grid_ctas"]
