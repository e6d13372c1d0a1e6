"""All priors of a model in one call: slices of full, partial and uneven runs, lists without slices, forces and totals against
float64 autograd over the differentiable terms."""
import pytest
import torch

import mlcg_b200
from helpers import prior_setup, random_walk_chain
from mlcg_b200 import nn as bnn
from mlcg_b200.nn.prior import _evaluate_together, _pair_slices

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n,B", [(5, 1), (10, 3), (20, 64), (36, 2), (37, 5), (38, 1), (100, 7), (130, 2), (133, 3), (134, 1), (270, 6)])
def test_forces_and_totals(n, B, dtype):
    data, priors = prior_setup(n, B, 4, torch.Generator().manual_seed(n))
    with torch.no_grad():
        priors["repulsion"].sigma.copy_(0.5 * (priors["repulsion"].sigma + priors["repulsion"].sigma.t()))
    gen = torch.Generator().manual_seed(n)      # (beads that do not overlap: the sums are fixed point)
    data.pos = torch.cat([random_walk_chain(n, gen, min_dist=3.0) for _ in range(B)]).to(dtype)
    data, priors = data.to(DEV), {k: p.to(DEV).eval() for k, p in priors.items()}
    assert (priors["repulsion"]._cached_list(data)[4] is not None) == (n >= 20)
    pos = data.pos.double().requires_grad_(True)
    for deterministic in (True, False):
        bnn.set_prior_determinism(deterministic)
        try:
            each, energy, forces = _evaluate_together(list(priors.values()), data, forces=True)
        finally:
            bnn.set_prior_determinism(True)
        tol = 1e-5 if dtype == torch.float32 else 1e-9
        e_sum, f_sum = 0.0, 0.0
        for k, p in priors.items():
            nl = data.neighbor_list[k]
            y = p._energy_terms(pos, nl["index_mapping"], p._params(data).double())
            want = torch.zeros(B, dtype=torch.float64, device=DEV).index_add_(0, nl["mapping_batch"], y)
            f = -torch.autograd.grad(want.sum(), pos)[0]
            assert torch.allclose(each[k][0].double(), want.detach(), rtol=tol, atol=tol), k
            assert float((each[k][1].double() - f).abs().max()) <= tol * (1 + float(f.abs().max())), k
            e_sum, f_sum = e_sum + want.detach(), f_sum + f
        assert torch.allclose(energy.double(), e_sum, rtol=tol, atol=tol)
        assert float((forces.double() - f_sum).abs().max()) <= tol * (1 + float(f_sum.abs().max()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n,B", [(20, 3), (21, 40), (24, 2), (25, 1), (32, 5), (33, 70), (34, 3), (57, 4), (66, 2), (129, 1), (321, 3)])
def test_slices_at_the_ends_of_stages(n, B, dtype):
    """Sliced lists of bonds and of repulsion, every pair of a structure both ways: runs of n - 1 terms that end inside, at and behind a
    stage of the copies, cut into parts that get no stage, one, or many."""
    gen = torch.Generator().manual_seed(n)
    every = torch.cartesian_prod(torch.arange(n), torch.arange(n)).t()
    every = every[:, every[0] != every[1]]
    mapping = torch.cat([every + k * n for k in range(B)], dim=1)
    owner = torch.arange(B).repeat_interleave(every.shape[1])
    priors = {"bonds": bnn.HarmonicBonds({(0, 0): {"k": 0.3, "x_0": 9.0}}), "repulsion": bnn.Repulsion({(0, 0): {"sigma": 3.5}})}
    lists = {k: mlcg_b200.make_neighbor_list(k, 2, mapping, owner) for k in priors}
    data = mlcg_b200.AtomicData(pos=torch.cat([random_walk_chain(n, gen, min_dist=3.0) for _ in range(B)]).to(dtype), atom_types=torch.zeros(n * B, dtype=torch.long),
                                batch=torch.arange(B).repeat_interleave(n), n_atoms=torch.full((B,), n), neighbor_list=lists).to(DEV)
    priors = {k: p.to(DEV).eval() for k, p in priors.items()}
    assert all(p._cached_list(data)[4] is not None for p in priors.values())
    each = _evaluate_together(list(priors.values()), data, forces=True)[0]
    again = _evaluate_together(list(priors.values()), data, forces=True)[0]
    pos = data.pos.double().requires_grad_(True)
    # (float32: sums of n terms of the roundings that one term has, as above)
    tol = 1e-5 if dtype == torch.float32 else 1e-9
    for k, p in priors.items():
        y = p._energy_terms(pos, lists[k]["index_mapping"].to(DEV), p._params(data).double())
        want = torch.zeros(B, dtype=torch.float64, device=DEV).index_add_(0, owner.to(DEV), y)
        f = -torch.autograd.grad(want.sum(), pos)[0]
        assert torch.allclose(each[k][0].double(), want.detach(), rtol=tol, atol=tol), k
        assert float((each[k][1].double() - f).abs().max()) <= tol * (1 + float(f.abs().max())), k
        assert torch.equal(each[k][0], again[k][0]) and torch.equal(each[k][1], again[k][1]), k


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_priors_repeat_bit_by_bit(dtype):
    """Steps of pair terms are copied into places that have just been read: a copy that overtakes the reads shows up as terms of another step, now
    and then.  (Sums are integers by default: nothing else may differ.)"""
    data, priors = prior_setup(150, 20, 4, torch.Generator().manual_seed(5))
    with torch.no_grad():                     # (its list is sliced)
        priors["repulsion"].sigma.copy_(0.5 * (priors["repulsion"].sigma + priors["repulsion"].sigma.t()))
    data.pos = torch.cat([random_walk_chain(150, torch.Generator().manual_seed(k), min_dist=3.0) for k in range(20)]).to(dtype)
    data, priors = data.to(DEV), [p.to(DEV).eval() for p in priors.values()]
    step = lambda: _evaluate_together(priors, data, forces=True)[0]  # noqa: E731
    want, differs = {k: (v[0].clone(), v[1].clone()) for k, v in step().items()}, torch.zeros((), dtype=torch.int64, device=DEV)
    assert any(p._cached_list(data)[4] is not None for p in priors)
    for _ in range(1000):
        for k, v in step().items():
            differs += (v[0] != want[k][0]).any() | (v[1] != want[k][1]).any()
    assert int(differs) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n", [21, 60, 130])
def test_slices_beside_more_single_terms(n, dtype):
    """A sliced list of bonds among twenty beads of a structure, every pair both ways, and a repulsion list of every pair one way, which is not
    sliced: with more of the single terms than of the others they have a launch of their own (n above 29), else they share one."""
    B, gen = 5, torch.Generator().manual_seed(n)
    every = torch.cartesian_prod(torch.arange(20), torch.arange(20)).t()
    both, half = every[:, every[0] != every[1]], torch.combinations(torch.arange(n)).t()
    priors = {"bonds": bnn.HarmonicBonds({(0, 0): {"k": 0.3, "x_0": 9.0}}), "repulsion": bnn.Repulsion({(0, 0): {"sigma": 3.5}})}
    lists, owner = {}, {}
    for k, m in (("bonds", both), ("repulsion", half)):
        owner[k] = torch.arange(B).repeat_interleave(m.shape[1])
        lists[k] = mlcg_b200.make_neighbor_list(k, 2, torch.cat([m + b * n for b in range(B)], dim=1), owner[k])
    data = mlcg_b200.AtomicData(pos=torch.cat([random_walk_chain(n, gen, min_dist=3.0) for _ in range(B)]).to(dtype), atom_types=torch.zeros(n * B, dtype=torch.long),
                                batch=torch.arange(B).repeat_interleave(n), n_atoms=torch.full((B,), n), neighbor_list=lists).to(DEV)
    priors = {k: p.to(DEV).eval() for k, p in priors.items()}
    assert priors["bonds"]._cached_list(data)[4] is not None and priors["repulsion"]._cached_list(data)[4] is None
    each = _evaluate_together(list(priors.values()), data, forces=True)[0]
    again = _evaluate_together(list(priors.values()), data, forces=True)[0]
    pos, tol = data.pos.double().requires_grad_(True), 1e-5 if dtype == torch.float32 else 1e-9          # (as above)
    for k, p in priors.items():
        y = p._energy_terms(pos, lists[k]["index_mapping"].to(DEV), p._params(data).double())
        want = torch.zeros(B, dtype=torch.float64, device=DEV).index_add_(0, owner[k].to(DEV), y)
        f = -torch.autograd.grad(want.sum(), pos)[0]
        assert torch.allclose(each[k][0].double(), want.detach(), rtol=tol, atol=tol), k
        assert float((each[k][1].double() - f).abs().max()) <= tol * (1 + float(f.abs().max())), k
        assert torch.equal(each[k][0], again[k][0]) and torch.equal(each[k][1], again[k][1]), k


def test_a_sliced_list_is_kept_once():
    """The slices of a pair list take the place of the 32-bit list and of the gathered parameters: 6 bytes a term and the padding."""
    data, priors = prior_setup(150, 20, 4, torch.Generator().manual_seed(3))
    gen = torch.Generator().manual_seed(3)      # (beads that do not overlap, as above)
    data.pos = torch.cat([random_walk_chain(150, gen, min_dist=3.0) for _ in range(20)]).float()
    p = priors["repulsion"]
    with torch.no_grad():
        p.sigma.copy_(0.5 * (p.sigma + p.sigma.t()))
    data, p = data.to(DEV), p.to(DEV).eval()
    M = data.neighbor_list["repulsion"]["index_mapping"].shape[1]
    before = torch.cuda.memory_allocated()
    assert p._cached_list(data)[4] is not None
    kept = torch.cuda.memory_allocated() - before
    assert 6 * M <= kept <= 1.3 * 6 * M
    together, alone = _evaluate_together([p], data, forces=True)[0]["repulsion"], bnn.GradientsOut(p, "forces").eval()(data).out["repulsion"]
    # (float32 sums of up to 300 terms in two orders: the bar of the test above, on both sides)
    assert torch.allclose(together[0], alone["energy"], rtol=2e-5, atol=2e-5)
    assert float((together[1] - alone["forces"]).abs().max()) <= 2e-5 * (1 + float(alone["forces"].abs().max()))


def test_lists_a_kernel_could_not_read_are_refused():
    data, priors = prior_setup(40, 2, 4, torch.Generator().manual_seed(4))
    with torch.no_grad():
        priors["repulsion"].sigma.copy_(0.5 * (priors["repulsion"].sigma + priors["repulsion"].sigma.t()))
    on_host = data.neighbor_list["repulsion"]["index_mapping"]
    data, p = data.to(DEV), priors["repulsion"].to(DEV).eval()
    _evaluate_together([p], data, forces=True)
    batch, data.batch = data.batch, data.batch[:-1]
    with pytest.raises(ValueError, match="one entry per bead"):
        _evaluate_together([p], data, forces=True)
    data.batch, data.neighbor_list["repulsion"]["index_mapping"] = batch, on_host
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        _evaluate_together([p], data, forces=True)


def test_pair_slices_of_beads_that_lie_far_apart():
    near = torch.arange(9, device=DEV, dtype=torch.int32)
    pairs = torch.stack([torch.zeros_like(near), near + 65535 - 8] ).repeat(1, 20)
    pairs[0] = torch.arange(20, device=DEV, dtype=torch.int32).repeat_interleave(9)
    params = torch.arange(180.0, device=DEV).view(1, -1)
    slices, beads, offsets, packed = _pair_slices(pairs, params)
    assert slices.tolist() == [[0, 3, 65527, 8]] and beads[0].tolist() == list(range(20)) + [-1] * 12
    assert packed[0, :, 3].flatten().tolist() == list(range(27, 36)) + [0.0] * 3
    assert offsets[:, 3].flatten().tolist() == list(range(9)) + [0] * 3 and int(offsets[:, 20:].to(torch.int32).max()) == 0
    pairs[1, 0] = 65527 + 65535
    assert _pair_slices(pairs, params) is not None
    pairs[1, 0] = 65528 + 65536
    assert _pair_slices(pairs, params) is None


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("beads,B", [(2, 1), (9, 1), (33, 2), (46, 1), (64, 33), (180, 3)])
def test_lists_made_from_tables(beads, B, dtype):
    """Indices, parameters, run starts and the comparison with the reversed list of one pass (chunks of 2048 terms), for complete pair
    lists, and for those with a term lost, doubled, replaced or of another parameter than its reverse."""
    from mlcg_b200.backend import get_backend
    be, gen, n = get_backend(), torch.Generator().manual_seed(beads), beads * B
    i = torch.arange(beads)
    one = torch.cartesian_prod(i, i).t()
    one = one[:, one[0] != one[1]]
    pairs = torch.cat([one + b * beads for b in range(B)], dim=1).to(DEV)
    M = pairs.shape[1]
    types = torch.randint(0, 5, (n,), generator=gen).to(DEV)
    table = torch.rand(5, 5, generator=gen, dtype=dtype).to(DEV)
    even, odd = table + table.t(), table
    idx, params, symmetric, starts = be.prior_list(pairs, types, [even, even * 2], None, n, True)
    assert torch.equal(idx.long(), pairs) and torch.equal(params, torch.stack([even[types[pairs[0]], types[pairs[1]]] * f for f in (1, 2)]))
    assert symmetric and (starts is None) == (beads < 9)
    if starts is not None:
        assert torch.equal(starts, torch.arange(0, M, beads - 1, device=DEV))
        slices, where, offsets, packed = _pair_slices(idx, params, starts)
        first = slices[:, 0].tolist()
        for run in (0, 31, 32, n - 1):
            if run < n:
                w, lane = run // 32, run % 32
                rows = slice(first[w], first[w] + int(slices[w, 1]))
                assert int(where[w, lane]) == run
                got = offsets[rows, lane].flatten()[: beads - 1].long() + int(slices[w, 2])
                assert torch.equal(got, pairs[1, run * (beads - 1): (run + 1) * (beads - 1)])
                assert torch.equal(packed[:, rows, lane].flatten(1)[:, : beads - 1], params[:, run * (beads - 1): (run + 1) * (beads - 1)])
    assert be.prior_list(pairs, types, None, params, n, True)[2]
    if len(torch.unique(types)) > 1 and beads > 2:
        assert not be.prior_list(pairs, types, [odd], None, n, True)[2]
        for at in (0, M // 2, M - 1):
            broken = pairs.clone()
            broken[:, at] = broken[:, at - 1]                      # one term lost, another one twice
            assert not be.prior_list(broken, types, [even], None, n, True)[2]
            given = params.clone()
            given[0, at] = given[0, at] * 1.5
            assert not be.prior_list(pairs, types, None, given, n, True)[2]
    for order in (3, 4):
        terms = torch.randint(0, n, (order, 2049), generator=gen).to(DEV)
        tables = [torch.rand(*([5] * order), generator=gen, dtype=dtype).to(DEV) for _ in range(3)]
        idx, params, symmetric, starts = be.prior_list(terms, types, tables, None, n, False)
        assert torch.equal(idx.long(), terms) and not symmetric and starts is None
        assert torch.equal(params, torch.stack([t[tuple(types[terms[o]] for o in range(order))] for t in tables]))
    be.check_pending()


def test_a_bead_that_does_not_exist_is_reported():
    from mlcg_b200.backend import get_backend
    be = get_backend()
    types, table = torch.zeros(4, dtype=torch.int64, device=DEV), torch.ones(1, 1, device=DEV)
    idx, _, symmetric, _ = be.prior_list(torch.tensor([[0, 1, 4, 2], [1, 0, 2, 4]], device=DEV), types, [table], None, 4, True)
    assert idx.tolist() == [[0, 1, -1, 2], [1, 0, 2, -1]]
    status = be._sticky_status(torch.device(DEV))
    assert int(status[0]) & 2
    status.zero_()


@pytest.mark.parametrize("there,missing", [(36, 64), (33, 31), (100, 1), (0, 64)])
def test_run_starts_of_a_list_for_a_longer_chain(there, missing):
    """A complete pair list over beads of which the last ones do not exist: as many run starts as runs are counted, and each where the
    written list has one (looked at on the host before anything reads through them); no slices."""
    from mlcg_b200.backend import get_backend
    be, n = get_backend(), there + missing
    i = torch.arange(n)
    pairs = torch.cartesian_prod(i, i).t()
    pairs = pairs[:, pairs[0] != pairs[1]].contiguous().to(DEV)
    types, table = torch.zeros(max(there, 1), dtype=torch.int64, device=DEV), torch.ones(1, 1, device=DEV)
    idx, params, symmetric, starts = be.prior_list(pairs, types, [table], None, there, True)
    first = idx[0].cpu()
    assert torch.equal(first, torch.where(pairs[0] < there, pairs[0], -1).cpu().to(torch.int32))
    heads = [0] + (torch.nonzero(first[1:] != first[:-1]).flatten() + 1).tolist()
    assert symmetric and starts.tolist() == heads and len(heads) == there + 1
    assert _pair_slices(idx, params, starts) is None
    status = be._sticky_status(torch.device(DEV))
    assert int(status[0]) & 2
    status.zero_()


@pytest.mark.parametrize("order,pairs", [(2, True), (2, False), (3, False), (4, False)])
def test_types_that_end_before_the_beads_do(order, pairs):
    """Beads past the end of the types are reported and left out; nothing is looked up behind the types."""
    from mlcg_b200.backend import get_backend
    be, n, typed = get_backend(), 40, 7
    mapping = torch.randint(0, typed, (order, 500), generator=torch.Generator().manual_seed(order)).to(DEV)
    mapping[order - 1, 100:] = torch.arange(400, device=DEV) % n
    types = torch.zeros(n, dtype=torch.int64, device=DEV)[:typed].clone()
    tables = [torch.full((1,) * order, 3.0, device=DEV)]
    idx, params, _, _ = be.prior_list(mapping, types, tables, None, n, pairs)
    assert torch.equal(idx.long(), torch.where(mapping < typed, mapping, -1)) and torch.equal(params, torch.full_like(params, 3.0))
    status = be._sticky_status(torch.device(DEV))
    assert int(status[0]) & 2
    status.zero_()


@pytest.mark.parametrize("name", ["bonds", "angles", "dihedrals", "repulsion"])
def test_lists_for_other_data_are_refused(name):
    """A list for a longer chain than the data, and beads of a type that the tables do not have: an error at the first call and at the
    next one, and the list is made again, whole, for data that fit."""
    data, priors = prior_setup(40, 2, 4, torch.Generator().manual_seed(4))
    data, p = data.to(DEV), priors[name].to(DEV).eval()
    data.pos = torch.cat([random_walk_chain(40, torch.Generator().manual_seed(5), min_dist=3.0) for _ in range(2)]).float().to(DEV)
    want, pos, batch, types = _evaluate_together([p], data, forces=True)[0][name], data.pos, data.batch, data.atom_types
    from mlcg_b200.backend import get_backend
    status = get_backend()._sticky_status(torch.device(DEV))
    for other in ((pos[:60], batch[:60], types), (pos, batch, types[:60]), (pos, batch, torch.where(torch.arange(80, device=DEV) == 70, 4, types))):
        data.pos, data.batch, data.atom_types = other
        for _ in range(2):
            with pytest.raises(IndexError, match="does not exist"):
                _evaluate_together([p], data, forces=True)
        data.pos, data.batch, data.atom_types = pos, batch, types
        got = _evaluate_together([p], data, forces=True)[0][name]
        assert all(torch.equal(a, b) for a, b in zip(got, want)) and int(status[0]) == 0
