"""GPU parity: the sm_100a kernels against the CPU oracle, bit for bit.

Every kernel rounds each product and sum once (explicitly rounded intrinsics), like the oracle
compiled without contraction, so the bar is bit-exact for every dtype pair and alpha/beta - stricter
than the <= 1 ulp the contracted reference would allow.
"""
import numpy as np
import pytest

import kernel_sim
import oracle
from helpers import (assert_bitexact, make_inputs, split, ttc_cases, uniform, NP, buffer_len)

pytestmark = pytest.mark.gpu


def _torch():
    import torch
    return torch


def run_gpu(A, B, perm, size, dtype, alpha, beta, lda=None, ldb=None, tuning=None, offset=0):
    """Runs the library on copies of A and B; offset shifts both buffers by elements (alignment)."""
    torch = _torch()
    from ttc_b200 import Plan
    ta, tb = split(dtype)
    tmap = {"s": torch.float32, "d": torch.float64, "c": torch.complex64, "z": torch.complex128}
    dA = torch.empty(A.size + offset, dtype=tmap[ta], device="cuda")
    dB = torch.empty(B.size + offset + 64, dtype=tmap[tb], device="cuda")
    dA[offset:].copy_(torch.from_numpy(A))
    dB[offset:offset + B.size].copy_(torch.from_numpy(B))
    canary = torch.from_numpy(uniform(64, tb, 99))
    dB[offset + B.size:].copy_(canary)
    plan = Plan(perm, size, dtype, complex(beta) != 0, lda, ldb, tuning)
    plan(dA[offset:], dB[offset:], alpha, beta)
    torch.cuda.synchronize()
    out = dB[offset:offset + B.size].cpu().numpy()
    tail = dB[offset + B.size:].cpu().numpy()
    assert np.array_equal(tail.view(np.uint8), canary.numpy().view(np.uint8)), "write past the end of B"
    desc = plan.describe()
    assert plan.wait_timeouts() == 0, "a stage wait of the bulk-copy kernel ran out of time"
    plan.close()
    return out, desc


def check_case(perm, size, dtype, alpha, beta, lda=None, ldb=None, tuning=None, seed=7, offset=0):
    A, B = make_inputs(size, perm, dtype, seed, lda, ldb)
    want = oracle.transpose(A, B.copy(), perm, size, alpha, beta, lda, ldb, dtype)
    got, desc = run_gpu(A, B, perm, size, dtype, alpha, beta, lda, ldb, tuning, offset)
    assert_bitexact(got, want, f"perm={perm} size={size} dtype={dtype} a={alpha} b={beta} lda={lda} "
                               f"ldb={ldb} tuning={tuning} plan={desc}")
    return desc


def test_ttc_reference_case_matrix():
    """The reference's own sweep (test-framework/ttc_test.py:80-217) on the GPU path."""
    for perm, size, dtype, alpha, beta in ttc_cases():
        check_case(perm, size, dtype, alpha, beta)


def test_against_ttc_golden_fixtures():
    """The GPU path against the outputs of TTC's own generated reference loop (tests/golden)."""
    import json
    from pathlib import Path
    z = np.load(Path(__file__).resolve().parent / "golden" / "ttc_reference_loop.npz")
    cases = json.loads(bytes(z["meta"]).decode())["cases"]
    for k, c in enumerate(cases):
        A, B = make_inputs(c["size"], c["perm"], c["dtype"], c["seed"], c["lda"], c["ldb"])
        for tuning in (None, {"tile_variant": 1}, {"tile_variant": 2}):
            got, desc = run_gpu(A, B, c["perm"], c["size"], c["dtype"], c["alpha"], c["beta"], c["lda"], c["ldb"],
                                tuning)
            assert_bitexact(got, z[f"B{k}"], f"golden {k} {c} tuning={tuning} plan={desc}")


def test_readme_shape_full_size():
    """perm 1,0,2 / 1000x768x16 fp32, alpha = beta = 1 (the README example)."""
    desc = check_case([1, 0, 2], [1000, 768, 16], "s", 1.0, 1.0)
    assert desc["kernel"] == "tile"
    check_case([1, 0, 2], [1000, 768, 16], "s", 1.0, 0.0)


@pytest.mark.parametrize("dtype,alpha", [("zc", complex(0.5, 0.25)), ("ds", 0.5), ("z", complex(0.5, 0.25)),
                                         ("d", 0.5)])
def test_strided_mixed_precision_config(dtype, alpha):
    """rank-4 perm 3,1,0,2, extents 96,80,72,64, lda = extents + {8,0,4,0}, B dense, beta = 0."""
    check_case([3, 1, 0, 2], [96, 80, 72, 64], dtype, alpha, 0.0, lda=[104, 80, 76, 64])


@pytest.mark.parametrize("dtype", ["s", "d", "c", "z", "sd", "ds", "cz", "zc"])
def test_padded_lda_ldb_and_complex_beta(dtype):
    ta, tb = split(dtype)
    cplx = ta in "cz"
    alpha = complex(1.25, -0.75) if cplx else 1.25
    beta = complex(-0.5, 0.3) if cplx else -0.5
    check_case([2, 0, 3, 1], [13, 9, 6, 11], dtype, alpha, beta, lda=[16, 10, 6, 12], ldb=[6, 15, 12, 9])
    check_case([1, 2, 0], [33, 17, 9], dtype, alpha, 0.0, ldb=[17, 12, 33])


TUNINGS = [{"vec": 1}, {"loop_order": 1}, {"loop_order": 2}, {"loop_order": 3}, {"blocks": 7}, {"tile_elems": 512},
           {"tile_elems": 8192}, {"run_bytes": 128}, {"run_bytes": 2048}, {"kernel": 1}, {"streaming": -1},
           {"streaming": 1}, {"round_robin": 1}, {"stages": 3}, {"stages": 7}, {"ctas_per_sm": 1},
           {"stages": 6, "ctas_per_sm": 2}, {"round_robin": 1, "blocks": 5}, {"round_robin": -1},
           {"round_robin": -1, "blocks": 5}, {"round_robin": -1, "claim_group": 3},
           {"round_robin": -1, "claim_group": 8, "blocks": 3}, {"bulk_copies": 1}, {"bulk_copies": 1, "round_robin": -1},
           {"bulk_copies": 1, "shifted_runs": 1}, {"lane_map": 1}]


@pytest.mark.parametrize("tuning", TUNINGS, ids=[str(t) for t in TUNINGS])
def test_schedule_knobs_do_not_change_results(tuning):
    for perm, size in ([[1, 0, 2], [300, 257, 5]], [[2, 0, 1], [7, 3, 20001]], [[0, 2, 1], [40, 33, 17]],
                       [[4, 2, 0, 3, 1], [9, 11, 7, 13, 5]], [[0, 1], [1000, 77]]):
        for dtype, beta in (("s", 0.0), ("d", 1.5), ("c", 0.0)):
            try:
                check_case(perm, size, dtype, 1.5, beta, tuning=tuning)
            except Exception as e:  # a forced tile kernel may not apply to every problem
                if "TTCB_ERR_UNSUPPORTED" in str(e) and tuning.get("kernel"):
                    continue
                raise


@pytest.mark.parametrize("order", [[0, 1, 2], [0, 2, 1], [1, 0, 2], [1, 2, 0], [2, 0, 1], [2, 1, 0]])
def test_every_explicit_loop_order(order):
    """TTC's --loopPerm as the tile grid's raster: each of the six orders of a rank-3 problem whose
    tile leaves every dimension in the grid, with ragged blocks, for beta = 0 and beta != 0."""
    for dtype, beta in (("s", 0.0), ("d", -0.5)):
        desc = check_case([1, 0, 2], [301, 263, 7], dtype, 1.5, beta, tuning={"raster": order})
        assert desc["loop_order"] == 4


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_misaligned_pointers_fall_back_to_narrow_accesses(offset):
    check_case([1, 0, 2], [64, 96, 3], "s", 1.0, 0.5, offset=offset)
    check_case([0, 2, 1], [256, 7, 9], "s", 2.0, 0.0, offset=offset)
    check_case([1, 0], [40, 33], "d", 1.0, 1.0, offset=offset)


def test_random_problems_ranks_1_to_6():
    rng = np.random.default_rng(11)
    for it in range(120):
        r = int(rng.integers(1, 7))
        size = [int(x) for x in rng.integers(1, 14, r)]
        perm = [int(x) for x in rng.permutation(r)]
        dtype = ["s", "d", "c", "z", "sd", "ds", "cz", "zc"][it % 8]
        beta = [0.0, 1.0, -0.5][it % 3]
        lda = [s + int(rng.integers(0, 2)) for s in size] if it % 4 == 0 else None
        check_case(perm, size, dtype, 1.5, beta, lda=lda, seed=it)


def test_edge_values_and_signed_zero():
    """Values that expose sign, rounding and special-value handling (NaN, inf, -0, denormals)."""
    torch = _torch()
    perm, size = [1, 0], [37, 41]
    for dtype in ("s", "d", "ds", "sd"):
        ta, tb = split(dtype)
        A, B = make_inputs(size, perm, dtype, 3)
        special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-40, -1e-310, 3.4e38, 1.0 + 2**-23],
                           dtype=np.float64)
        A[: special.size] = special.astype(A.dtype)
        B[-special.size:] = special.astype(B.dtype)
        for alpha, beta in ((1.0, 0.0), (-1.0, 1.0), (3.0, -2.0)):
            want = oracle.transpose(A, B.copy(), perm, size, alpha, beta, dtype=dtype)
            got, _ = run_gpu(A, B, perm, size, dtype, alpha, beta)
            assert_bitexact(got, want, f"special {dtype} {alpha} {beta}")


def test_empty_and_single_element():
    check_case([0], [1], "s", 2.0, 1.0)
    check_case([1, 0], [1, 1], "z", complex(2, 1), 0.0)
    from ttc_b200 import Plan
    torch = _torch()
    p = Plan([1, 0], [0, 5], "s")
    x = torch.zeros(4, device="cuda")
    p(x, x, 1.0)  # no-op
    torch.cuda.synchronize()


def test_error_paths_do_not_poison_the_context():
    import ctypes
    from ttc_b200 import Plan, TTCError
    from ttc_b200._native import check, lib
    torch = _torch()
    x = torch.zeros(64, device="cuda")
    y = torch.zeros(64, device="cuda")
    p0 = Plan([1, 0], [8, 8], "s", beta_nonzero=False)
    with pytest.raises(TTCError) as e:
        p0(x, y, 1.0, 0.5)  # beta given to a plan made for beta == 0
    assert e.value.code == "TTCB_ERR_BETA"
    with pytest.raises(TTCError) as e:
        Plan([1, 0], [8, 8], "s", lda=[4, 8])
    assert e.value.code == "TTCB_ERR_BAD_LD"
    with pytest.raises(TTCError) as e:
        Plan([0, 0], [8, 8], "s")
    assert e.value.code == "TTCB_ERR_BAD_PERM"
    al = (ctypes.c_float * 1)(1.0)
    with pytest.raises(TTCError) as e:  # A not aligned to its element size
        check(lib().ttcb_transpose(p0.handle, x.data_ptr() + 2, y.data_ptr(), ctypes.cast(al, ctypes.c_void_p),
                                   None, None))
    assert e.value.code == "TTCB_ERR_ALIGN"
    p1 = Plan([1, 0], [8, 8], "s", beta_nonzero=True)
    with pytest.raises(TTCError) as e:  # beta missing for a beta != 0 plan
        check(lib().ttcb_transpose(p1.handle, x.data_ptr(), y.data_ptr(), ctypes.cast(al, ctypes.c_void_p),
                                   None, None))
    assert e.value.code == "TTCB_ERR_BETA"
    # the context is still healthy
    check_case([1, 0], [8, 8], "s", 1.0, 0.0)


def test_torch_permute_agrees_on_large_sweep_shapes():
    """Size-independent property at full size: for alpha = 1, beta = 0 the result is a pure
    permutation, identical to torch.permute(...).contiguous() bit for bit."""
    torch = _torch()
    from ttc_b200 import Plan
    import ttc_b200.workloads as wl
    cases = wl.sweep_cases(seed=2024)[:6]
    rasters, edges = set(), 0
    for c in cases:
        size, perm = c["size"], c["perm"]
        tdt = torch.float32 if c["dtype"] == "s" else torch.float64
        n = int(np.prod(size))
        A = torch.rand(n, dtype=tdt, device="cuda") * 2 - 1
        B = torch.empty_like(A)
        p = Plan(perm, size, c["dtype"], False)
        p(A, B, 1.0, 0.0)
        # A viewed row-major with reversed dims; B's dims are A's dims in perm order
        At = A.view(*reversed(size))
        nd = len(size)
        want = At.permute(*[nd - 1 - perm[j] for j in reversed(range(nd))]).contiguous().view(-1)
        torch.cuda.synchronize()
        assert torch.equal(B, want), (perm, size, p.describe())
        d = p.describe()
        rasters.add(d["loop_order"])
        edges += bool(d.get("edges"))
        del A, B, At, want
        torch.cuda.empty_cache()
    # the planner's raster choice (B-major for short B runs) and edge plans are both exercised
    assert rasters == {1, 3} and edges > 0, (rasters, edges)


@pytest.mark.parametrize("perm,size", [([1, 0], [46341, 46341]), ([2, 0, 1], [3, 65537, 10923])])
def test_more_than_2_to_the_31_elements(perm, size):
    """Maximum sizes: tensors with more than 2^31 elements (8.6 GB each in fp32) need 64-bit tile
    bases (TTC used int everywhere). alpha = 1, beta = 0 is a pure permutation, compared with
    torch.permute(...).contiguous() bit for bit on the GPU."""
    torch = _torch()
    from ttc_b200 import Plan
    n = int(np.prod(size))
    assert n > 2**31
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    A = torch.rand(n, device="cuda", generator=g)
    B = torch.empty_like(A)
    p = Plan(perm, size, "s", False)
    p(A, B, 1.0, 0.0)
    nd = len(size)
    want = A.view(*reversed(size)).permute(*[nd - 1 - perm[j] for j in reversed(range(nd))]).contiguous().view(-1)
    torch.cuda.synchronize()
    assert torch.equal(B, want), (perm, size, p.describe())
    p.close()
    del A, B, want
    torch.cuda.empty_cache()


@pytest.mark.parametrize("ragged", [0, 1])
@pytest.mark.parametrize("dtype,beta", [("s", 0.0), ("d", -0.5), ("zc", 0.0)])
def test_ragged_tiles_beside_the_staged_kernel_streams_and_graphs(dtype, beta, ragged):
    """Prime extents leave ragged last blocks: the staged kernel moves the complete tiles while the
    side stream, forked from the caller's stream and joined back, moves the rest - as edge plans
    (the ragged boxes planned as transpositions of their own, offset into A and B) or, with the
    `ragged` knob at 1, with the element-wise ragged-tile kernel. The result must equal the oracle
    when called on the default stream, on a side torch stream, and when the call is captured into
    a CUDA graph and replayed (the fork and join are captured with it)."""
    torch = _torch()
    from ttc_b200 import Plan
    perm, size = [2, 0, 1], [67, 131, 251]
    ta, tb = split(dtype)
    tmap = {"s": torch.float32, "d": torch.float64, "c": torch.complex64, "z": torch.complex128}
    A, B = make_inputs(size, perm, dtype, 31)
    want = oracle.transpose(A, B.copy(), perm, size, 1.5, beta, dtype=dtype)
    plan = Plan(perm, size, dtype, beta != 0, tuning={"ragged": ragged})
    d = plan.describe()
    t = d["tile"]
    assert t["async"] == 1 and t["ragged_tiles"] > 0, t
    assert bool(d.get("edges")) == (ragged == 0), d
    dA = torch.from_numpy(A).cuda()
    for mode in ("default", "stream", "graph"):
        dB = torch.from_numpy(B.copy()).cuda()
        if mode == "default":
            plan(dA, dB, 1.5, beta)
        elif mode == "stream":
            s = torch.cuda.Stream()
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                plan(dA, dB, 1.5, beta, s)
            torch.cuda.current_stream().wait_stream(s)
        else:
            g = torch.cuda.CUDAGraph()
            s = torch.cuda.Stream()
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                with torch.cuda.graph(g, stream=s):
                    plan(dA, dB, 1.5, beta, s)
            dB.copy_(torch.from_numpy(B))
            g.replay()
        torch.cuda.synchronize()
        assert_bitexact(dB.cpu().numpy(), want, f"{mode} {dtype} beta={beta} tile={t}")
    plan.close()


@pytest.mark.parametrize("offset", [0, 1])
def test_edge_plans_random_ragged_problems(offset):
    """Problems whose tiles leave ragged last blocks (prime extents), with padded lda/ldb, a unit
    first dimension with a padded leading dimension (the edge boxes then start with a unit
    dimension), mixed and complex types, beta != 0 and misaligned base pointers: the edge plans
    (offset sub-problems moved by the staged kernel on the side stream) must give the oracle's
    result bit for bit."""
    rng = np.random.default_rng(23 + offset)
    primes = [3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 67]
    with_edges = 0
    for it in range(48):
        r = int(rng.integers(2, 6))
        size = [int(rng.choice(primes)) for _ in range(r)]
        perm = [int(x) for x in rng.permutation(r)]
        while perm == sorted(perm):
            perm = [int(x) for x in rng.permutation(r)]
        lda = ldb = None
        if it % 3 == 1:
            lda = [s + int(rng.integers(0, 3)) for s in size]
            ldb = [size[perm[j]] + int(rng.integers(0, 3)) for j in range(r)]
        if it % 4 == 2:
            size, perm = [1] + size, [0] + [x + 1 for x in perm]
            lda = [2] + (lda or size[1:])
            ldb = [1] + (ldb or [size[perm[j]] for j in range(1, r + 1)])
        dtype = ["s", "d", "zc", "ds", "c"][it % 5]
        beta = [0.0, -0.5][it % 2]
        tuning = {"tile_elems": [0, 256, 512][it % 3]} if it % 3 else None
        desc = check_case(perm, size, dtype, 1.5, beta, lda, ldb, tuning, seed=100 + it, offset=offset)
        with_edges += bool(desc.get("edges"))
    assert with_edges >= 12, with_edges


# problems whose ragged tiles are too many for the staged kernel's own launch: one ragged dimension or two
EDGE_PLANS = [("s", -0.5, [1, 0, 2], [131, 131, 257], 512, 2), ("d", -0.5, [3, 0, 2, 1], [37, 37, 37, 67], 0, 1),
              ("c", 0.0, [1, 0, 2, 3], [41, 13, 5, 1021], 512, 1), ("z", 1.2, [1, 0, 3, 2], [37, 7, 131, 67], 256, 1),
              ("zc", 0.0, [1, 0, 3, 2], [37, 7, 41, 163], 256, 1), ("sd", -0.5, [1, 0, 3, 2], [97, 31, 67, 17], 8192, 1)]


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("dtype,beta,perm,size,tile_elems,boxes", EDGE_PLANS)
def test_edge_plans_on_streams_in_graphs_and_batches(dtype, beta, perm, size, tile_elems, boxes, offset):
    """Ragged tiles that edge plans move: the plan says that its own launch does not move them, and the
    result is the oracle's bit for bit on the default stream, on a side stream, replayed from a captured
    graph and as a problem of a batch, from aligned and misaligned pointers."""
    torch = _torch()
    from ttc_b200 import Plan
    from ttc_b200.batched import Batch
    A, B = make_inputs(size, perm, dtype, 41)
    want = oracle.transpose(A, B.copy(), perm, size, 1.5, beta, dtype=dtype)
    plan = Plan(perm, size, dtype, beta != 0, tuning={"tile_elems": tile_elems})
    d = plan.describe()
    assert d["tile"]["ragged_inline"] == 0 and len(d["edges"]) == boxes and all("plan" in e for e in d["edges"]), d
    dA = torch.from_numpy(np.concatenate([A[:offset], A])).cuda()[offset:]
    room = torch.empty(offset + B.size + 8, dtype=torch.from_numpy(B).dtype, device="cuda")
    dB = room[offset:offset + B.size]
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        plan(dA, dB, 1.5, beta, side)
    batch = Batch([plan], [dA], [dB], alpha=1.5, beta=beta)

    def on_side():
        with torch.cuda.stream(side):
            plan(dA, dB, 1.5, beta, side)

    for what, call in (("default", lambda: plan(dA, dB, 1.5, beta)), ("stream", on_side), ("graph", graph.replay),
                       ("batch", batch.launch), ("batch graph", lambda: batch.launch(graph=True))):
        room.fill_(3.0)
        dB.copy_(torch.from_numpy(B))
        torch.cuda.synchronize()
        call()
        torch.cuda.synchronize()
        assert_bitexact(dB.cpu().numpy(), want, f"{what} {dtype} {d['tile']}")
        assert bool((room[offset + B.size:] == 3.0).all()) and bool((room[:offset] == 3.0).all()), what
    batch.close()
    del graph
    plan.close()


def test_plans_that_move_ragged_tiles_in_their_own_launch_have_no_edge_plans():
    """Their description lists the boxes that the ragged tiles cover, without plans; the same boxes that
    the edge plans of ragged tiles would have."""
    _torch()
    from ttc_b200 import Plan
    for perm, size in [([2, 0, 1], [67, 131, 251]), ([1, 0], [65, 129]), ([2, 0, 1], [67, 31, 53])]:
        plan = Plan(perm, size, "s", False)
        d = plan.describe()
        assert d["tile"]["ragged_inline"] > 0 and d["edges"], d
        boxes = kernel_sim.edge_boxes(perm, size, "s", False)
        assert d["edges"] == [{"offA": b["offA"], "offB": b["offB"]} for b in boxes]
        plan.close()


@pytest.mark.parametrize("dtype,beta", [("s", 0.0), ("s", -0.5), ("d", 0.0), ("d", -0.5), ("c", 1.2), ("zc", 0.0),
                                        ("sd", -0.5)])
def test_ragged_tiles_in_the_staged_launch(dtype, beta):
    """Ragged tiles that the staged kernel moves in its own launch: one ragged dimension or two,
    remainders of one element, of all but one and of whole vectors, limits on and off the vector grid,
    misaligned pointers, claimed tiles, shifted runs, bulk copies and deep rings, bit for bit against the
    oracle; and the same launch captured and replayed."""
    seen = set()
    for perm, size in [([1, 0], [65, 129]), ([1, 0], [127, 95]), ([1, 0, 2], [36, 68, 5]), ([1, 0], [100, 412]),
                       ([2, 1, 0], [11, 2, 1093]), ([2, 0, 1], [67, 31, 53]), ([0, 2, 1], [3, 97, 61]),
                       ([1, 2, 0], [26, 653, 8]), ([3, 1, 0, 2], [17, 3, 7, 29])]:
        for tuning in ({"tile_elems": 512}, {"tile_elems": 1024, "round_robin": -1, "blocks": 5},
                       {"tile_elems": 1024, "shifted_runs": 1}, {"tile_elems": 2048, "bulk_copies": 1, "stages": 6}):
            for offset in (0, 1):
                desc = check_case(perm, size, dtype, 1.5, beta, tuning=tuning, offset=offset)
                t = desc.get("tile") or {}
                seen.add((t.get("ragged_inline"), t.get("shifted_runs"), t.get("bulk")))
    assert {k[0] for k in seen} >= {1, 2}, seen


@pytest.mark.parametrize("dtype", ["s", "sd", "ds"])
def test_tiles_of_eight_narrow_accesses_per_thread(dtype):
    """Problems large enough (64 MB moved) for tiles of up to eight 4-byte accesses per thread on a side,
    with odd extents that leave such accesses on A, on B or on both, ragged tiles, misaligned pointers,
    round-robin and claimed tiles, bit for bit against the oracle (beta = 0; with beta the same shapes keep
    four)."""
    wide = 0
    for perm, size in [([1, 0], [27, 300007]), ([1, 0], [300011, 27]), ([1, 0, 2], [99, 17, 4813]),
                       ([2, 1, 0], [10, 25, 32771])]:
        for offset, beta, tuning in ((0, 0.0, None), (1, 0.0, None), (0, 0.0, {"round_robin": -1}), (0, -0.5, None)):
            desc = check_case(perm, size, dtype, 1.5, beta, tuning=tuning, offset=offset)
            t = desc["tile"]
            narrow = max(t["P"] // desc["vecA"], t["P"] // desc["vecB"])
            if t["reg"] == 1:  # (tiles off the register path may be larger)
                assert narrow <= (2048 if beta == 0 else 1024), desc
                wide += narrow > 1024
    assert wide >= 3, wide


def test_claimed_tiles_with_concurrent_launches_and_slot_reuse():
    """The staged kernel's tiles claimed from the plan's counters: one plan launched on four streams
    at once (different counter slots), then 150 launches in a row on one stream (every slot used and
    reset more than twice), each result bit for bit equal to the oracle's."""
    import torch
    from ttc_b200 import Plan
    perm, size = [2, 0, 1], [67, 45, 311]
    plan = Plan(perm, size, "s", True, tuning={"blocks": 16, "round_robin": -1})
    assert plan.describe()["tile"]["async"] == 1 and plan.describe()["tile"]["claims"] == 1
    n = int(np.prod(size))
    streams = [torch.cuda.Stream() for _ in range(4)]
    ins, outs, wants = [], [], []
    for k in range(4):
        A, B = make_inputs(size, perm, "s", 300 + k)
        wants.append(oracle.transpose(A, B.copy(), perm, size, 1.5, -0.5, dtype="s"))
        ins.append(torch.from_numpy(A).cuda())
        outs.append(torch.from_numpy(B).cuda())
    torch.cuda.synchronize()
    for k, st in enumerate(streams):
        plan(ins[k], outs[k], 1.5, -0.5, st)
    torch.cuda.synchronize()
    for k in range(4):
        assert_bitexact(outs[k].cpu().numpy(), wants[k], f"stream {k}")
    A, B = make_inputs(size, perm, "s", 400)
    want = B.copy()
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    for rep in range(150):
        plan(dA, dB, 1.0, 0.5)
        oracle.transpose(A, want, perm, size, 1.0, 0.5, dtype="s")
    torch.cuda.synchronize()
    assert_bitexact(dB.cpu().numpy(), want, "150 launches")
    plan.close()


def test_large_plans_in_turn_and_in_a_row_see_each_others_results():
    """Launches of different and of the same plans behind each other on one stream, each reading what the one
    before wrote, below and above the size from which a launch lets the next one begin beside it only when
    it repeats its plan: bit for bit torch's permutations."""
    torch = _torch()
    from ttc_b200 import Plan

    def permuted(t, perm):  # t: row-major view of the column-major tensor
        n = t.dim()
        return t.permute(*[n - 1 - perm[j] for j in reversed(range(n))]).contiguous()

    steps = [[2, 0, 1], [2, 0, 1], [1, 0, 2]]
    for mb in (40, 130):
        size = [96, 160, mb * 1_000_000 // 8 // (96 * 160)]
        x = torch.rand(*reversed(size), device="cuda")
        wants, plans = [x], []
        for perm in steps:
            plans.append(Plan(perm, list(reversed(wants[-1].shape)), "s", False))
            wants.append(permuted(wants[-1], perm))
        outs = [x] + [torch.empty_like(x) for _ in steps]
        for repeat in (1, 1, 3, 2, 1):
            for y in outs[1:]:
                y.fill_(float("nan"))
            for p, src, dst in zip(plans, outs, outs[1:]):
                for _ in range(repeat):
                    p(src, dst)
            torch.cuda.synchronize()
            for k, (y, w) in enumerate(zip(outs[1:], wants[1:])):
                assert torch.equal(y.view(-1), w.view(-1)), (mb, repeat, k)
        for p in plans:
            p.close()


@pytest.mark.parametrize("perm,size,dtype,beta,claims,group", [
    ([1, 0, 2], [1000, 768, 16], "s", 1.0, 0, 2),            # 98 MB of tensors
    ([1, 0, 2], [1024, 768, 25], "s", 0.0, 0, 2),            # 157 MB
    ([1, 0, 2], [1024, 768, 26], "s", 0.0, 1, 2),            # 164 MB
    ([1, 0], [27, 1941807], "s", -0.5, 0, 4),                # thin, with beta: A by 16 bytes, B by 4
    ([2, 0, 1], [13, 2016492, 2], "s", -0.5, 0, 4),          # tiles of 12 KiB, runs of 2 and 4 KB
    ([1, 0], [7489829, 7], "s", 0.0, 1, 2),                  # of 14 KiB, runs of 1 and 7 KB, A by 4 bytes
    ([1, 0, 2], [1565, 1155, 29], "s", -0.5, 1, 4),          # of 12 KiB, runs of 128 bytes
    ([5, 2, 1, 3, 0, 4], [10, 7, 13, 11, 81, 65], "s", 0.0, 1, 4),  # of 7 KiB, runs of 280 and 52 bytes
    ([5, 4, 0, 2, 1, 3], [7, 11, 16, 38, 5, 112], "d", -0.5, 1, 2)])  # of 29 KB
def test_planners_claim_rule(perm, size, dtype, beta, claims, group):
    """Tiles are claimed by default for tensors past L2, by twos or, of tiles under 13 KiB, by fours, but not small
    tiles with long runs on both sides nor thin matrices with beta; the autotuner's mirror of the rule says
    the same."""
    _torch()
    from ttc_b200 import Plan
    from ttc_b200.autotune import Problem, staged_claims
    plan = Plan(perm, size, dtype, beta != 0)
    d = plan.describe()
    assert (d["tile"]["claims"], d["tile"]["claim_group"]) == (claims, group), d
    assert staged_claims(Problem(perm, size, dtype, 1.0, beta), {}, d) == bool(claims), d
    plan.close()


@pytest.mark.parametrize("group", [7, 8, 9, 12, 13, 16, 63, 64, 100])
def test_claims_of_any_group_size(group):
    """Claims of up to 64 consecutive tiles (more count as 64), decoded in batches of the largest divisor up to
    eight: bit for bit against the oracle with few CTAs, which then claim many groups, and many, for the
    shallowest and the deepest ring, by plain and by bulk copies."""
    for blocks in (3, 0):
        for tuning in ({"stages": 3}, {"stages": 7}, {"bulk_copies": 1}):
            for size in ([67, 45, 311], [64, 48, 16]):
                desc = check_case([2, 0, 1], size, "s", 1.5, -0.5,
                                  tuning=dict(tuning, claim_group=group, round_robin=-1, blocks=blocks, tile_elems=256))
                assert desc["tile"]["claims"] == 1 and desc["tile"]["claim_group"] == min(group, 64), desc


def test_claimed_tiles_of_overlapping_launches_have_their_own_counters():
    """Launches of one plan that run at the same time never share a tile counter, however many launches lie
    between them: one held back on a stream until 64 launches later, one replayed from a CUDA graph beside
    a direct one, and one on each of 70 streams; each result bit for bit
    equal to the oracle's."""
    import torch
    from ttc_b200 import Plan
    perm, size = [2, 0, 1], [67, 45, 311]
    plan = Plan(perm, size, "s", False, tuning={"blocks": 16, "round_robin": -1, "tile_elems": 256})
    assert plan.describe()["tile"]["claims"] == 1
    A, B = make_inputs(size, perm, "s", 300)
    want = oracle.transpose(A, B, perm, size, 1.5, 0.0, dtype="s")
    src = torch.from_numpy(A).cuda()
    dst = [torch.empty_like(src) for _ in range(70)]
    gate, s1, s2, s3 = (torch.cuda.Stream() for _ in range(4))

    def together(*calls):
        """Starts the calls at the same time, each on a stream of its own."""
        for d in dst:
            d.fill_(float("nan"))
        torch.cuda.synchronize()
        with torch.cuda.stream(gate):
            torch.cuda._sleep(20_000_000)
            opened = gate.record_event()
        for st, call in calls:
            if st is not s3:
                st.wait_event(opened)
            with torch.cuda.stream(st):
                call()
        torch.cuda.synchronize()

    def check(used, what):
        for k in used:
            assert_bitexact(dst[k].cpu().numpy(), want, f"{what}, output {k}")

    between = lambda: [plan(src, dst[2], 1.5, 0.0, s3) for _ in range(63)]
    for rep in range(4):
        together((s1, lambda: plan(src, dst[0], 1.5, 0.0, s1)), (s3, between),
                 (s2, lambda: plan(src, dst[1], 1.5, 0.0, s2)))
        check((0, 1, 2), "64 launches apart")
    graphs = []
    for rep in range(4):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s1):
            plan(src, dst[0], 1.5, 0.0, s1)
        graphs.append(g)
        together((s1, g.replay), (s3, between), (s2, lambda: plan(src, dst[1], 1.5, 0.0, s2)))
        check((0, 1, 2), "a replay beside a launch")
    together(*[(torch.cuda.Stream(), lambda k=k: plan(src, dst[k], 1.5, 0.0)) for k in range(70)])
    check(range(70), "70 streams")
    del graphs
    plan.close()


SHIFTED = [([1, 0], [99, 1001]), ([1, 0, 3, 2], [99, 17, 35, 3]), ([1, 0, 2], [45, 77, 9]),
           ([2, 1, 0], [10, 25, 2097]), ([0, 2, 1], [31, 110, 15]), ([2, 0, 1], [23, 13, 240])]


BULK = [([1, 0, 2], [300, 256, 5]), ([2, 0, 1], [8, 64, 1000]), ([1, 0], [1024, 999]), ([3, 1, 0, 2], [16, 20, 24, 9]),
        ([1, 0, 2], [1000, 768, 16])]


@pytest.mark.parametrize("dtype", ["s", "d", "c", "z", "sd", "ds", "zc"])
def test_bulk_a_copies(dtype):
    """A runs moved by one bulk copy each (cp.async.bulk into the stage, an mbarrier per stage):
    bit for bit against the oracle for aligned runs and for shifted runs at A offsets of 0 to 3
    elements, beta = 0 and beta != 0, round-robin and claimed tiles, the shallowest and deepest rings;
    no stage wait runs out of time (run_gpu checks the plan's count)."""
    used = 0
    for perm, size in BULK + SHIFTED:
        for beta in (0.0, -0.5):
            desc = check_case(perm, size, dtype, 1.5, beta, tuning={"bulk_copies": 1})
            used += int((desc.get("tile") or {}).get("bulk", 0))
            for offset in (0, 1, 3):
                check_case(perm, size, dtype, 1.5, beta, offset=offset, tuning={"bulk_copies": 1, "shifted_runs": 1})
            check_case(perm, size, dtype, 1.5, beta, tuning={"bulk_copies": 1, "round_robin": 1, "stages": 3})
            check_case(perm, size, dtype, 1.5, beta, tuning={"bulk_copies": 1, "blocks": 9, "stages": 7,
                                                             "round_robin": -1})
    assert used > 0


LANE_MAPS = [([1, 0, 2, 3], [48, 3, 48, 29]), ([1, 0], [54, 48]), ([2, 3, 1, 0], [17, 22, 53, 12]), ([1, 0], [32, 20]),
             ([1, 2, 0], [18, 31, 58]), ([1, 0], [4, 58]), ([2, 1, 0], [40, 48, 30]), ([1, 2, 3, 0], [29, 54, 59, 29])]


@pytest.mark.parametrize("dtype", ["s", "d", "c", "sd", "ds"])
def test_lane_maps(dtype):
    """Plans whose register path takes B vectors from several B runs per warp (lane_map = 1: maps
    the planner picks against the gather's bank conflicts, in natural or A-sorted run order),
    including maps whose last footprint row reaches past the tile's runs: bit for bit against the
    oracle for beta = 0 and beta != 0, with claimed tiles, bulk copies and round-robin tiles."""
    used = 0
    for perm, size in LANE_MAPS:
        for beta in (0.0, -0.5):
            desc = check_case(perm, size, dtype, 1.5, beta, tuning={"lane_map": 1})
            used += int((desc.get("tile") or {}).get("lane_map", 0) > 0)
            check_case(perm, size, dtype, 1.5, beta, tuning={"lane_map": 1, "round_robin": -1, "blocks": 7})
            check_case(perm, size, dtype, 1.5, beta, tuning={"lane_map": 1, "bulk_copies": 1})
            check_case(perm, size, dtype, 1.5, beta, tuning={"lane_map": 1, "round_robin": 1, "stages": 5})
    assert used > 0


def test_bounded_wait_gives_up_and_the_context_survives():
    """The stage wait of the bulk-copy kernel has a time limit: on a barrier phase that nothing
    completes it gives up after the limit and reports it, and the context stays usable; on a phase
    that completes it does not give up."""
    import ctypes
    import time
    from ttc_b200 import _native
    lib = _native.lib()
    n = ctypes.c_uint(7)
    t0 = time.perf_counter()
    assert lib.ttcb_test_bounded_wait(20_000_000, 0, ctypes.byref(n)) == 0
    assert n.value == 1 and time.perf_counter() - t0 >= 0.02
    assert lib.ttcb_test_bounded_wait(20_000_000, 1, ctypes.byref(n)) == 0
    assert n.value == 0
    check_case([1, 0, 2], [300, 256, 5], "s", 1.5, -0.5, tuning={"bulk_copies": 1})


@pytest.mark.parametrize("dtype", ["s", "d", "c", "sd", "ds", "cz"])
def test_shifted_a_runs(dtype):
    """A runs of odd lengths and offsets copied as the 16-byte chunks that cover them, shifted per
    tile (and by A's own misalignment, offsets of 1 to 3 elements): bit for bit against the oracle,
    for beta = 0 and beta != 0, and equal to the plain layout (shifted_runs = -1)."""
    used = 0
    for perm, size in SHIFTED:
        for beta in (0.0, -0.5):
            for offset in (0, 1, 3):
                desc = check_case(perm, size, dtype, 1.5, beta, offset=offset, tuning={"shifted_runs": 1})
                used += int((desc.get("tile") or {}).get("shifted_runs", 0))
            check_case(perm, size, dtype, 1.5, beta, tuning={"shifted_runs": -1})
            check_case(perm, size, dtype, 1.5, beta, tuning={"shifted_runs": 1, "round_robin": 1, "stages": 5})
            check_case(perm, size, dtype, 1.5, beta, tuning={"shifted_runs": 1, "blocks": 9, "round_robin": -1})
    assert used > 0
