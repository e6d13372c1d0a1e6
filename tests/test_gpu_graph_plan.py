"""The radius graph with its pair plan: the bit-mask route of small batches and the cell route give the same lists and plans as the
separate entry points and the oracle, at and around the sizes where the routes meet."""
import numpy as np
import pytest
import torch

from mlcg_b200.backend import get_backend
from oracle import radius_ref

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("sizes", [[1], [2], [31, 0, 33], [10] * 64, [73], [385], [2048], [2047, 1], [2049], [1] * 2000 + [40], [400, 700, 900, 300], [768, 769, 767, 5, 1200], [4600, 4601, 10, 385], [8192, 5000],
                                   [8300, 300], [8300] + [20] * 60, [100] * 30])
def test_plan_with_the_graph(sizes, dtype):
    rng = np.random.default_rng(len(sizes) + sizes[0])
    ptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    pos = (rng.random((int(ptr[-1]), 3)) * max(sizes) ** (1 / 3) * 2.0).astype(dtype)
    be = get_backend()
    t = torch.as_tensor(pos, device=DEV)
    for given in ("ptr", "n_atoms"):
        more = dict(n_atoms=torch.as_tensor(sizes, dtype=torch.int64, device=DEV)) if given == "n_atoms" else {}
        res = be.radius_graph(t, None if more else torch.as_tensor(ptr, device=DEV), 4.0, 1000, False, 1, want_distance=True, want_plan=True, **more)
        assert torch.equal(res["ptr"].cpu(), torch.as_tensor(ptr))
        want = radius_ref.radius_graph_c(pos, ptr, 4.0, 1000, False, "cluster")
        assert torch.equal(res["edge_index"].cpu(), torch.from_numpy(want))
        assert torch.equal(torch.stack([res["row0"], res["row1"]]).long(), res["edge_index"])
        assert torch.equal(res["mapping_batch"].cpu(), torch.as_tensor(np.repeat(np.arange(len(sizes)), sizes))[res["edge_index"][0].cpu()])
        if want.shape[1] == 0:
            assert res["twin"] is None
            continue
        twin, sel, pair_of, status = be.pair_plan(res["row0"], res["row1"], res["offsets"], len(pos), fresh_status=True)
        assert int(status[0]) == 0
        assert torch.equal(res["twin"], twin) and torch.equal(res["sel"], sel) and torch.equal(res["pair_of"], pair_of)
    be.check_pending()


@pytest.mark.parametrize("n,loop,rule,cap", [(300, False, 1, 7), (300, False, 0, 7), (300, True, 1, 9), (2048, False, 1, 20), (40, True, 0, 1000)])
def test_neighbour_caps_and_loops(n, loop, rule, cap):
    rng = np.random.default_rng(n + cap)
    pos = (rng.random((n, 3)) * n ** (1 / 3) * 1.5).astype(np.float32)
    ptr = np.array([0, n // 3, n], dtype=np.int64)
    res = get_backend().radius_graph(torch.as_tensor(pos, device=DEV), torch.as_tensor(ptr, device=DEV), 3.0, cap, loop, rule, want_plan=True)
    want = radius_ref.radius_graph_c(pos, ptr, 3.0, cap, loop, "cluster" if rule else "native")
    assert torch.equal(res["edge_index"].cpu(), torch.from_numpy(want))
    assert bool(res["status"] & 1) == (cap < 100)
    assert (res["twin"] is None) == (loop or cap < 100)


@pytest.mark.parametrize("n", [200, 3000])
@pytest.mark.parametrize("room", [0.5, 1.0, 1.3])
def test_fixed_capacity(n, room):
    rng = np.random.default_rng(n)
    pos = torch.as_tensor((rng.random((n, 3)) * n ** (1 / 3) * 2).astype(np.float32), device=DEV)
    ptr = torch.tensor([0, n], device=DEV)
    be = get_backend()
    ref = be.radius_graph(pos, ptr, 4.0, 1000, False, 1, want_plan=True)
    E = ref["row0"].numel()
    cap = int(E * room) // 2 * 2
    res = be.graph_capacity(pos, ptr, None, 4.0, 1000, cap, torch.zeros((2, cap), dtype=torch.int32, device=DEV))
    live = min(E, cap)
    assert res["counts"].tolist() == [live, live // 2]
    if room < 1.0:
        with pytest.raises(RuntimeError):
            be.check_pending()
        assert int(res["offsets"].max()) == cap and 0 <= int(res["twin"][:live].min()) and int(res["twin"][:live].max()) < cap
        return
    be.check_pending()
    assert torch.equal(res["offsets"], ref["offsets"])
    for k in ("row0", "row1", "twin", "pair_of"):
        assert torch.equal(res[k][:live], ref[k]), k
    assert torch.equal(res["sel"][:live // 2], ref["sel"])


def test_counts_read_by_several_threads():
    """Each host thread reads its own counts from the line that its graph's kernels write, on its own stream."""
    from concurrent.futures import ThreadPoolExecutor
    be = get_backend()
    rng = np.random.default_rng(5)
    work = []
    for n in (50, 700, 3000, 41, 2100, 900):
        pos = (rng.random((n, 3)) * n ** (1 / 3) * 2).astype(np.float32)
        ptr = np.array([0, n // 2, n], dtype=np.int64)
        work.append((torch.as_tensor(pos, device=DEV), torch.as_tensor(ptr, device=DEV), radius_ref.radius_graph_c(pos, ptr, 4.0, 1000, False, "cluster").shape[1]))
    torch.cuda.synchronize()

    def run(k):
        stream, got = torch.cuda.Stream(), []
        with torch.cuda.device(0), torch.cuda.stream(stream):
            for i in range(60):
                pos, ptr, want = work[(i * (k + 1) + k) % len(work)]
                got.append(be.radius_graph(pos, ptr, 4.0, 1000, False, 1, want_plan=True)["edge_index"].shape[1] == want)
        stream.synchronize()
        return all(got)

    with ThreadPoolExecutor(4) as pool:
        assert all(pool.map(run, range(4)))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("sizes", [[3, 0, 5] * 400, [0] * 40 + [768] * 3 + [0] * 3, [1] * 2100, [2] * 1025, [767, 768, 768], [64, 31, 33] * 1100, [700] * 3 + [769], [1000, 600, 500, 1],
                                   [0] * 40 + [1024] * 3 + [0] * 3, [1023, 1024, 1024, 33], [900] * 3 + [1025]])
def test_bit_rows_of_whole_batches(sizes, dtype):
    """Batches of structures that all fit a bit row are counted and scanned in three launches (structures found by a warp among 1, 32, 33 and
    more boundaries, parts of 32 points, blocks of 1024); one larger structure sends the batch the other way."""
    rng = np.random.default_rng(len(sizes) + sizes[0])
    ptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    assert 2048 < ptr[-1] <= 1024 * len(sizes)
    pos = (rng.random((int(ptr[-1]), 3)) * max(sizes) ** (1 / 3) * 2.0).astype(dtype)
    be, t = get_backend(), torch.as_tensor(pos, device=DEV)
    want = radius_ref.radius_graph_c(pos, ptr, 4.0, 1000, False, "cluster")
    for given in (dict(ptr=torch.as_tensor(ptr, device=DEV)), dict(ptr=None, n_atoms=torch.as_tensor(sizes, dtype=torch.int64, device=DEV))):
        res = be.radius_graph(t, given.pop("ptr"), 4.0, 1000, False, 1, want_distance=True, want_plan=True, **given)
        assert torch.equal(res["ptr"].cpu(), torch.as_tensor(ptr)) and res["status"] == 0
        assert torch.equal(res["edge_index"].cpu(), torch.from_numpy(want))
        if want.shape[1]:
            twin, sel, pair_of, status = be.pair_plan(res["row0"], res["row1"], res["offsets"], len(pos), fresh_status=True)
            assert int(status[0]) == 0
            assert torch.equal(res["twin"], twin) and torch.equal(res["sel"], sel) and torch.equal(res["pair_of"], pair_of)
    for loop, rule, cap in ((True, 1, 1000), (False, 1, 3), (False, 0, 3)):
        res = be.radius_graph(t, torch.as_tensor(ptr, device=DEV), 4.0, cap, loop, rule)
        cut = radius_ref.radius_graph_c(pos, ptr, 4.0, cap, loop, "cluster" if rule else "native")
        assert torch.equal(res["edge_index"].cpu(), torch.from_numpy(cut))
        # (the cluster rule counts the point itself among its cap + 1: a list is cut short where it lost somebody)
        assert bool(res["status"] & 1) == (cut.shape[1] < want.shape[1] + (len(pos) if loop else 0))
    be.check_pending()


@pytest.mark.parametrize("sizes", [[1] * 1500 + [700] * 2, [700] * 2 + [1] * 1500, [3] * 17 + [1000] * 2 + [0] * 60, [24] * 31 + [0] * 33 + [25] * 60, [100] * 30 + [0] * 300])
def test_structures_far_from_where_their_points_suggest(sizes):
    """The look at the 32 boundaries around a point's share of the batch: structures before, behind and outside of them."""
    test_bit_rows_of_whole_batches(sizes, np.float32)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("r", [0.55, 0.7, 0.9, 2.0])
@pytest.mark.parametrize("sizes", [[31, 32, 33, 64], [2000], [100] * 25, [33, 31] * 40, [1000, 900, 300], [1024, 65, 1024]])
def test_rows_of_words_from_half_full_to_full(sizes, r, dtype):
    """Rows with so many hits in a word that they are written word by word, rows just below, and both kinds in one row's words: edges, plans and rows
    cut inside a word, against the oracle.  (Points of a unit cube; at 2 every pair.)"""
    rng = np.random.default_rng(len(sizes))
    ptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    pos = rng.random((int(ptr[-1]), 3)).astype(dtype)
    be, t, p = get_backend(), torch.as_tensor(pos, device=DEV), torch.as_tensor(ptr, device=DEV)
    batch = torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes)).to(DEV)
    want = torch.from_numpy(radius_ref.radius_graph_c(pos, ptr, r, 2000, False, "cluster"))
    res = be.radius_graph(t, p, r, 2000, False, 1, want_distance=True, want_plan=True)
    assert torch.equal(res["edge_index"].cpu(), want)
    twin, sel, pair_of, status = be.pair_plan(res["row0"], res["row1"], res["offsets"], len(pos), fresh_status=True)
    assert int(status[0]) == 0 and torch.equal(res["twin"], twin) and torch.equal(res["sel"], sel) and torch.equal(res["pair_of"], pair_of)
    for loop, cap in ((False, 2000), (True, 2000), (False, 45), (True, 17)):
        cut = torch.from_numpy(radius_ref.radius_graph_c(pos, ptr, r, cap, loop, "cluster"))
        assert torch.equal(be.radius_graph(t, p, r, cap, loop, 1, want_plan=False)["edge_index"].cpu(), cut)
        if len(pos) <= 2048:
            assert torch.equal(be.radius_graph_small(t, batch, r, cap, loop, 1)["edge_index"].cpu(), cut)
    be.check_pending()


@pytest.mark.parametrize("how", ["rows shuffled", "rows reversed", "cut in the middle", "upper halves alone", "other centres"])
def test_a_list_without_a_plan_is_reported_and_stays_inside(how):
    """mlcgb_pair_plan of lists that are not what it takes: status bit 2, and every entry is an index, none of it outside the arrays."""
    be, n, gen = get_backend(), 300, torch.Generator().manual_seed(3)
    pos = (torch.rand(n, 3, generator=gen) * 12).to(DEV)
    ref = be.radius_graph(pos, torch.tensor([0, n], device=DEV), 4.0, 1000, False, 1)
    row0, row1, offsets = ref["row0"].cpu(), ref["row1"].cpu(), ref["offsets"].cpu()
    ends = offsets.tolist()
    if how == "rows shuffled":
        row1 = torch.cat([row1[a:b][torch.randperm(b - a, generator=gen)] for a, b in zip(ends, ends[1:])])
    elif how == "rows reversed":
        row1 = torch.cat([row1[a:b].flip(0) for a, b in zip(ends, ends[1:])])
    elif how == "cut in the middle":
        keep = ends[n // 2] // 2 * 2
        row0, row1, offsets = row0[:keep], row1[:keep], offsets.clamp(max=keep)
    elif how == "upper halves alone":
        up = row0 < row1
        row0, row1 = row0[up], row1[up]
        offsets = torch.cat([torch.zeros(1, dtype=torch.int64), torch.bincount(row0.long(), minlength=n).cumsum(0)])
        if row0.numel() % 2:
            row0, row1, offsets = row0[:-1], row1[:-1], offsets.clamp(max=row0.numel() - 1)
    else:
        row0 = row0.flip(0)
    E = row0.numel()
    rows, offsets = torch.stack([row0, row1]).contiguous().to(DEV), offsets.to(DEV)
    guard, mark = 4096, -7
    sizes = (E, E // 2, E)
    bufs = [torch.full((guard + k + guard,), mark, dtype=torch.int32, device=DEV) for k in sizes]
    for b, k in zip(bufs, sizes):
        b[guard:guard + k] = 0
    status, wsb = torch.zeros(4, dtype=torch.int32, device=DEV), be.lib.mlcgb_pair_plan_workspace_bytes(n)
    ws = torch.empty(wsb, dtype=torch.uint8, device=DEV)
    assert be.lib.mlcgb_pair_plan(rows[0].data_ptr(), rows[1].data_ptr(), offsets.data_ptr(), E, n, ws.data_ptr(), wsb, *(b[guard:].data_ptr() for b in bufs),
                                  status.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    assert int(status[0]) & 4
    for b, k, most in zip(bufs, sizes, (E, E, E // 2)):
        inside = b[guard:guard + k]
        assert int(inside.min()) >= 0 and int(inside.max()) < most
        assert bool((b[:guard] == mark).all()) and bool((b[guard + k:] == mark).all())


@pytest.mark.parametrize("sizes", [[2], [31, 0, 33], [2048], [2049], [1] * 2000 + [60], [384, 385] * 30, [700] * 4, [768, 5, 0, 1200], [4600, 4601, 10, 385], [385] * 47, [385] * 48, [8192, 5000],
                                   [8193, 300], [8193] + [20] * 60, [100] * 30])
def test_plan_of_a_list_given_later(sizes):
    """The plan made of a list when it is first used is the one that the separate entry point gives, whatever the route to it."""
    from mlcg_b200 import radius_graph
    from mlcg_b200.autograd import plan_of
    from mlcg_b200.neighbor_list import radius_cuda
    gen, be, n = torch.Generator().manual_seed(len(sizes) + sizes[0]), get_backend(), sum(sizes)
    pos = (torch.rand(n, 3, generator=gen) * max(sizes) ** (1 / 3) * 2.0).to(DEV)
    batch = torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes)).to(DEV)
    ptr = torch.tensor([0] + sizes, device=DEV).cumsum(0)
    for edges in (radius_graph(pos, 4.0, batch, max_num_neighbors=1000, flow="target_to_source"), radius_cuda(pos, ptr, 4.0, 1000, True)[0]):
        plan = plan_of(edges, n)
        assert torch.equal(torch.stack([plan.row0, plan.row1]).long(), edges) and plan.symmetric
        if edges.shape[1] == 0:
            continue
        offsets = torch.cat([torch.zeros(1, dtype=torch.int64, device=DEV), torch.bincount(edges[0], minlength=n).cumsum(0)])
        twin, sel, pair_of, status = be.pair_plan(plan.row0.clone(), plan.row1.clone(), offsets, n, fresh_status=True)
        assert int(status[0]) == 0 and torch.equal(plan.ptr_out, offsets)
        assert torch.equal(plan.perm_in, twin) and torch.equal(plan.half_selection(), sel) and torch.equal(plan.pair_index(), pair_of)
        assert plan_of(edges, n) is plan
    be.check_pending()
    assert int(be._sticky_status(torch.device(DEV))[0]) == 0


@pytest.mark.parametrize("sizes", [[300], [400] * 60, [3000, 100]])
@pytest.mark.parametrize("how", ["shuffled", "another structure", "other centres", "no bead", "one named by all"])
def test_a_list_changed_behind_its_version_is_reported(sizes, how):
    """Writes that a list does not count (``.data``) before its plan is made: reported, and every entry of the plan is an index."""
    from mlcg_b200 import radius_graph
    from mlcg_b200.autograd import plan_of
    gen, be, n = torch.Generator().manual_seed(5), get_backend(), sum(sizes)
    pos = (torch.rand(n, 3, generator=gen) * max(sizes) ** (1 / 3) * 2.0).to(DEV)
    batch = torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes)).to(DEV)
    edges = radius_graph(pos, 4.0, batch, max_num_neighbors=1000, flow="target_to_source")
    E = edges.shape[1]
    if how == "shuffled":
        edges.data[1] = edges[1][torch.randperm(E, generator=gen).to(DEV)]
    elif how == "another structure":
        edges.data[1] = (edges[1] + sizes[0] // 2 + 1) % n
    elif how == "other centres":
        edges.data[0] = edges[0].flip(0)
    elif how == "no bead":
        edges.data[1, ::7] = n + 5
        edges.data[1, 3::7] = -1
    else:
        edges.data[1] = sizes[0] // 2
    status = be._sticky_status(torch.device(DEV))
    status.zero_()
    plan = plan_of(edges, n)
    assert int(status[0]) & 4
    status.zero_()
    for t, most in ((plan.row0, n), (plan.row1, n), (plan.perm_in, E), (plan.half_selection(), E), (plan.pair_index(), E // 2)):
        assert int(t.min()) >= 0 and int(t.max()) < most


@pytest.mark.parametrize("sizes", [[40, 30], [900, 900, 600], [1000, 1500, 700], [3000, 100], [20] * 150])
@pytest.mark.parametrize("given", ["one short", "many short", "one over", "far over", "one below zero", "one beyond all"])
def test_sizes_that_do_not_add_up(sizes, given):
    """``n_atoms`` of another batch, on every route of the graph: an error, and the call after it has its own result."""
    import mlcg_b200
    from mlcg_b200 import nn as bnn
    be, n, gen = get_backend(), sum(sizes), torch.Generator().manual_seed(2)
    pos = (torch.rand(n, 3, generator=gen) * max(sizes) ** (1 / 3) * 2.5).to(DEV)
    right = torch.tensor(sizes, device=DEV)
    wrong = right.clone()
    if given == "one short":
        wrong[-1] -= 1
    elif given == "many short":
        wrong = wrong // 3
    elif given == "one over":
        wrong[0] += 1
    elif given == "far over":
        wrong *= 1000
    elif given == "one below zero":
        wrong[-1] = -5
    else:
        wrong[0] = 2 ** 40
    torch.manual_seed(0)
    cut = bnn.CosineCutoff(0.0, 4.0)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 32, trainable=False), cut, [128], embedding_size=5, num_interactions=2).eval().to(DEV)
    model, types = bnn.GradientsOut(net, "forces").eval(), torch.zeros(n, dtype=torch.int64, device=DEV)
    data = lambda s: mlcg_b200.AtomicData(pos=pos.clone(), atom_types=types, batch=torch.repeat_interleave(torch.arange(len(sizes), device=DEV), right), n_atoms=s)  # noqa: E731
    graph = lambda s: be.radius_graph(pos, None, 4.0, 1000, False, 1, n_atoms=s, want_plan=True)  # noqa: E731
    want, out = graph(right), model(data(right)).out["SchNet"]
    with pytest.raises(ValueError, match="does not add up"):
        graph(wrong)
    for as_given in (wrong, wrong.to(torch.int32), wrong.repeat_interleave(2)[::2]):
        if int(as_given.sum()) == n:
            continue                                    # (2^40 as int32)
        with pytest.raises(ValueError, match="does not add up"):
            model(data(as_given))
    bnn.set_edge_capacity(model, want["row0"].numel() * 2)
    with pytest.raises(ValueError, match="does not add up"):
        model(data(wrong))
        be.check_pending()
    fixed = model(data(right)).out["SchNet"]
    be.check_pending()
    bnn.set_edge_capacity(model, None)
    got, again = graph(right), model(data(right)).out["SchNet"]
    be.check_pending()
    assert torch.equal(got["edge_index"], want["edge_index"]) and torch.equal(got["twin"], want["twin"])
    assert torch.equal(again["energy"], out["energy"]) and torch.equal(again["forces"], out["forces"])
    assert torch.allclose(fixed["energy"], out["energy"], rtol=1e-5, atol=1e-5 * float(out["energy"].abs().max()))


@pytest.mark.parametrize("sizes", [[300], [73] * 60])
def test_a_plan_asked_for_on_another_stream(sizes):
    """The list goes out of use while the stream that makes its plan is still behind: its memory is not given to others before."""
    from mlcg_b200 import radius_graph
    from mlcg_b200.autograd import plan_of
    gen, be, n = torch.Generator().manual_seed(8), get_backend(), sum(sizes)
    pos = (torch.rand(n, 3, generator=gen) * 9).to(DEV)
    batch = torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes)).to(DEV)
    make = lambda: radius_graph(pos, 4.0, batch, max_num_neighbors=1000, flow="target_to_source")  # noqa: E731
    want_edges = make().clone()
    want = plan_of(make(), n)
    want = [t.clone() for t in (want.row0, want.row1, want.ptr_out, want.perm_in, want.half_selection(), want.pair_index())]
    side = torch.cuda.Stream()
    for _ in range(3):
        edges = make()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            torch.cuda._sleep(20_000_000)                  # (about 10 ms)
            plan = plan_of(edges, n)
        sizes_held = [edges.numel() * 8, (n + 1) * 8, (len(sizes) + 1) * 8]
        del edges
        held = [torch.full((k,), 0x7f, dtype=torch.uint8, device=DEV) for k in sizes_held for _ in range(4)]
        torch.cuda.synchronize()
        got = (plan.row0, plan.row1, plan.ptr_out, plan.perm_in, plan.half_selection(), plan.pair_index())
        assert all(torch.equal(a, b) for a, b in zip(got, want)) and len(held) == 12
        del plan, got, held
    assert torch.equal(make(), want_edges)
    be.check_pending()


@pytest.mark.parametrize("n", [300, 3000, 9000])
@pytest.mark.parametrize("how", ["last first", "shuffled", "below zero", "size too small", "size too large"])
def test_batch_vectors_that_are_not_sorted(n, how):
    """Undefined neighbours, but of points that are there: boundaries that ascend from 0 to N, edges inside it, and a call after it that is right."""
    from mlcg_b200 import radius_graph
    gen, be = torch.Generator().manual_seed(n), get_backend()
    pos = (torch.rand(n, 3, generator=gen) * n ** (1 / 3) * 1.5).to(DEV)
    sorted_batch = torch.sort(torch.randint(0, max(n // 700, 2), (n,), generator=gen))[0].to(DEV)
    want = radius_graph(pos, 3.0, sorted_batch, max_num_neighbors=1000)
    batch, more = sorted_batch.clone(), {}
    if how == "last first":
        batch = batch.flip(0)
    elif how == "shuffled":
        batch = batch[torch.randperm(n, generator=gen).to(DEV)]
    elif how == "below zero":
        batch -= 1
    else:
        more = dict(batch_size=int(batch.max()) + (0 if how == "size too small" else 5))
    ptr = be.batch_to_ptr(batch, more["batch_size"]) if more else be.batch_boundaries(batch)
    assert int(ptr[0]) == 0 and int(ptr[-1]) == n * (ptr.numel() > 1) and bool((ptr[1:] >= ptr[:-1]).all())
    if ptr.numel() > 1:
        edges = radius_graph(pos, 3.0, batch, max_num_neighbors=1000, **more)
        assert edges.numel() == 0 or (int(edges.min()) >= 0 and int(edges.max()) < n and not bool((edges[0] == edges[1]).any()))
    assert torch.equal(radius_graph(pos, 3.0, sorted_batch, max_num_neighbors=1000), want)
