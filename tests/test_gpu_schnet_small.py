"""Evaluations of fewer beads than one 128-row tile (single proteins, a bead or two) take the one-call route like any other."""
import pytest
import torch

import mlcg_b200
from mlcg_b200 import nn as bnn
from mlcg_b200.backend import get_backend

from helpers import random_walk_chain
from test_gpu_schnet import E_RTOL, F_ATOL, _oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("sizes", [[1], [2], [5, 1, 30], [73], [127], [128], [129]])
def test_batches_below_one_tile(sizes):
    gen = torch.Generator().manual_seed(sum(sizes))
    torch.manual_seed(1)
    upper, L, B = 10.0, 2, len(sizes)
    cut = bnn.CosineCutoff(0.0, upper)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 50, trainable=False), cut, [128], hidden_channels=128, embedding_size=6, num_filters=128,
                             num_interactions=L)
    pos = torch.cat([random_walk_chain(n, gen, jitter=0.2) for n in sizes])
    types_, batch = torch.randint(0, 6, (sum(sizes),), generator=gen), torch.arange(B).repeat_interleave(torch.tensor(sizes))
    e_x, f_x, _ = _oracle(net, "expnormal", upper, L, pos, types_, batch, B, torch.float64)
    net = net.to(DEV).eval()
    assert net._whole_model_setup(pos.to(DEV)) is not None
    out = bnn.GradientsOut(net, "forces").eval()(mlcg_b200.AtomicData(pos=pos.to(DEV), atom_types=types_.to(DEV), batch=batch.to(DEV),
                                                                      n_atoms=torch.tensor(sizes).to(DEV))).out["SchNet"]
    assert torch.allclose(out["energy"].cpu().double(), e_x, rtol=E_RTOL, atol=E_RTOL * float(e_x.abs().max()))
    assert float((out["forces"].cpu().double() - f_x).abs().max()) < F_ATOL


def test_evaluation_from_positions_keeps_up_with_changing_sizes():
    """One library call from positions: the workspace guess of one batch meets a denser, a larger and a smaller one, and a list
    without edges; the numbers are those of the evaluation on a given neighbour list."""
    torch.manual_seed(0)
    cut = bnn.CosineCutoff(0.0, 8.0)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 32, trainable=False), cut, [128], embedding_size=5, num_interactions=2).eval().to(DEV)
    model = bnn.GradientsOut(net, "forces").eval()
    gen = torch.Generator().manual_seed(3)
    for sizes, box in (([12, 9], 9.0), ([12, 9], 5.0), ([300, 41, 2], 14.0), ([2500], 30.0), ([4], 6.0), ([1], 1.0), ([2], 200.0)):
        n = sum(sizes)
        pos, types_ = torch.rand(n, 3, generator=gen).mul(box).to(DEV), torch.randint(0, 5, (n,), generator=gen).to(DEV)
        batch = torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes)).to(DEV)
        make = lambda: mlcg_b200.AtomicData(pos=pos.clone(), atom_types=types_, batch=batch, n_atoms=torch.tensor(sizes, device=DEV))  # noqa: E731
        got = model(make()).out["SchNet"]
        given = make()
        given.neighbor_list = net.neighbor_list(given, 8.0)
        want = model(given).out["SchNet"]
        assert torch.equal(got["energy"], want["energy"]) and torch.equal(got["forces"], want["forces"]), sizes


@pytest.mark.parametrize("sizes", [[2], [3, 1], [31, 33], [64] * 8, [1] * 1000 + [20], [1024, 1023], [2047], [2048], [1] * 2000 + [48], [2049], [1, 0, 4]])
def test_graph_made_inside_the_evaluation(sizes):
    """Up to 2048 beads the lists are made by the evaluation's first two launches, ahead of the host's look at the edge count or without
    one: the numbers are those of the evaluation on a given list, bit by bit, for workspaces that are too small, exact and larger;
    a list cut short leaves the route."""
    from mlcg_b200.backend import get_backend
    torch.manual_seed(0)
    cut = bnn.CosineCutoff(0.0, 6.0)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 32, trainable=False), cut, [128], embedding_size=5, num_interactions=2).eval().to(DEV)
    model, be, n = bnn.GradientsOut(net, "forces").eval(), get_backend(), sum(sizes)
    gen = torch.Generator().manual_seed(n)
    pos, types_ = (torch.rand(n, 3, generator=gen) * 2.5 * max(sizes) ** (1 / 3)).to(DEV), torch.randint(0, 5, (n,), generator=gen).to(DEV)
    batch = torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes)).to(DEV)
    make = lambda **kw: mlcg_b200.AtomicData(pos=pos.clone(), atom_types=types_, batch=batch, **kw)  # noqa: E731
    by_size = dict(n_atoms=torch.tensor(sizes, device=DEV))
    given = make(**by_size)
    given.neighbor_list = net.neighbor_list(given, 6.0)
    E = given.neighbor_list["SchNet"]["index_mapping"].shape[1]
    want = model(given).out["SchNet"]
    for guess in (0.0, (E - 2) / n / 1.04, E / n, 3 * E / n):
        for kw in (by_size, {}):
            net.__dict__["_mlcgb_edges_per_bead"] = max(guess, 0.0)
            got = model(make(**kw)).out["SchNet"]
            assert torch.equal(got["energy"], want["energy"]) and torch.equal(got["forces"], want["forces"]), guess
    for cap in (E, E + 2, 3 * E):
        bnn.set_edge_capacity(model, cap)
        got = model(make(**by_size)).out["SchNet"]
        be.check_pending()
        assert torch.equal(got["energy"], want["energy"]) and torch.equal(got["forces"], want["forces"]), cap
    bnn.set_edge_capacity(model, E - 2)
    if E > 2:
        model(make(**by_size))
        with pytest.raises(RuntimeError, match="capacity"):
            be.check_pending()
    bnn.set_edge_capacity(model, None)
    if max(sizes) > 8:
        net.max_num_neighbors = 3
        cut_short = model(make(**by_size)).out["SchNet"]
        given = make(**by_size)
        given.neighbor_list = net.neighbor_list(given, 6.0, 3)
        want = model(given).out["SchNet"]
        assert torch.equal(cut_short["energy"], want["energy"]) and torch.equal(cut_short["forces"], want["forces"])
    be.check_pending()


@pytest.mark.parametrize("sizes", [[40, 30], [2500]])
def test_weights_written_by_the_launch_before(sizes):
    """A call whose first kernels read weights sees what the kernel launched just before it wrote to them, and so does one product
    whose second operand the product before it has made."""
    from mlcg_b200.backend import get_backend
    torch.manual_seed(0)
    cut = bnn.CosineCutoff(0.0, 8.0)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 32, trainable=False), cut, [128], embedding_size=5, num_interactions=2).eval().to(DEV)
    model = bnn.GradientsOut(net, "forces").eval()
    n = sum(sizes)
    data = mlcg_b200.AtomicData(pos=torch.rand(n, 3, device=DEV).mul(20.0), atom_types=torch.zeros(n, dtype=torch.int64, device=DEV),
                                batch=torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes)).to(DEV), n_atoms=torch.tensor(sizes, device=DEV))
    data.neighbor_list = net.neighbor_list(data, 8.0)
    params = [p.data for p in net.parameters()]
    versions, want = [[p * s for p in params] for s in (1.0, 0.5, 1.5)], []
    write = lambda v: torch._foreach_copy_(params, v)  # noqa: E731
    for v in versions:
        write(v)
        torch.cuda.synchronize()
        want.append({k: t.clone() for k, t in model(data).out["SchNet"].items()})
    for k in [1, 0, 2] * 10:
        write(versions[k])
        got = model(data).out["SchNet"]
        assert torch.equal(got["forces"], want[k]["forces"]) and torch.equal(got["energy"], want[k]["energy"])
    be = get_backend()
    x, w = torch.randn(128, 128, device=DEV), torch.randn(128, 128, device=DEV) / 11
    y = be.gemm_fused(0, x, w)
    torch.cuda.synchronize()
    z = be.gemm_fused(0, x, y)
    for _ in range(20):
        assert torch.equal(be.gemm_fused(0, x, be.gemm_fused(0, x, w)), z)


def test_recordings_of_one_model_stand_by_themselves():
    """Two recordings and plain evaluations of one model over different data: the row buffers and the prior lists that a recording
    reads stay its own, and nothing of it writes memory that has been given back."""
    from helpers import prior_setup
    torch.manual_seed(0)
    cut = bnn.CosineCutoff(0.0, 9.0)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 32, trainable=False), cut, [128], embedding_size=4, num_interactions=2)
    sets = []
    for k, (n, B) in enumerate(((30, 6), (45, 5))):
        data, priors = prior_setup(n, B, 4, torch.Generator().manual_seed(k))
        gen = torch.Generator().manual_seed(k)
        data.pos = torch.cat([random_walk_chain(n, gen, min_dist=3.0) for _ in range(B)]).float()
        sets.append(data.to(DEV))
    with torch.no_grad():
        priors["repulsion"].sigma.copy_(0.5 * (priors["repulsion"].sigma + priors["repulsion"].sigma.t()))
    model = bnn.SumOut(torch.nn.ModuleDict({"SchNet": bnn.GradientsOut(net, "forces"), **{k: bnn.GradientsOut(p, "forces") for k, p in priors.items()}}))
    model = bnn.set_edge_capacity(model.eval().to(DEV), 9000)
    fresh = lambda d: mlcg_b200.AtomicData(pos=d.pos.clone(), atom_types=d.atom_types, batch=d.batch, n_atoms=d.n_atoms,  # noqa: E731
                                           neighbor_list={k: dict(v) for k, v in d.neighbor_list.items()})
    want = []
    for d in sets:
        out = model(fresh(d)).out
        want.append((out["energy"].clone(), out["forces"].clone()))
    fields = [mlcg_b200.GraphedForceField(model, fresh(d)) for d in sets]
    rows = [[v for v in f._kept[1] if isinstance(v, tuple) and len(v) == 2 and torch.is_tensor(v[1])] for f in fields]
    assert len(rows[0]) == len(rows[1]) == 1 and rows[0][0][1].data_ptr() != rows[1][0][1].data_ptr()
    model(fresh(sets[1]))
    junk = [torch.full((2, 9000), 7, dtype=torch.int32, device=DEV) for _ in range(64)] + [torch.full((2 ** 16,), 7, dtype=torch.int32, device=DEV) for _ in range(64)]
    for _ in range(2):
        for f, d, (e, g) in zip(fields, sets, want):
            got = f(d.pos)
            assert torch.equal(got[0], e) and torch.equal(got[1], g)
    fields[0].check()
    assert all(bool((j == 7).all()) for j in junk)


@pytest.mark.parametrize("sizes", [[73], [10] * 64, [268] * 8])
@pytest.mark.parametrize("blocks", [1, 2])
def test_positions_and_biases_written_in_place_between_evaluations(sizes, blocks):
    """One buffer of positions and one set of biases, overwritten between replays and between plain evaluations: kernels that start early
    read what lies there now, not what an evaluation before has left in a cache."""
    torch.manual_seed(blocks)
    cut = bnn.CosineCutoff(0.0, 9.0)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 32, trainable=False), cut, [128], embedding_size=4, num_interactions=blocks)
    model = bnn.GradientsOut(net.to(DEV), "forces").eval()
    n, gen = sum(sizes), torch.Generator().manual_seed(len(sizes))
    frames = [torch.cat([random_walk_chain(k, gen, min_dist=3.0) for k in sizes]).to(DEV) for _ in range(3)]
    biases = [[torch.randn(p.shape, generator=gen).mul(0.1).to(DEV) for name, p in net.named_parameters() if name.endswith("bias")] for _ in frames]
    here, kept = torch.empty(n, 3, device=DEV), [p for name, p in net.named_parameters() if name.endswith("bias")]
    batch = torch.arange(len(sizes), device=DEV).repeat_interleave(torch.tensor(sizes, device=DEV))
    make = lambda pos: mlcg_b200.AtomicData(pos=pos, atom_types=torch.arange(n, device=DEV) % 4, batch=batch, n_atoms=torch.tensor(sizes, device=DEV))  # noqa: E731

    def write(k):
        here.copy_(frames[k])
        with torch.no_grad():
            torch._foreach_copy_(kept, biases[k])

    want = []
    for k, frame in enumerate(frames):
        write(k)
        torch.cuda.synchronize()
        out = model(make(frame.clone())).out["SchNet"]
        want.append((out["energy"].clone(), out["forces"].clone()))
        torch.cuda.synchronize()
    field = None
    if n >= 128:                            # (the fewest beads that a recording takes)
        bnn.set_edge_capacity(model, 40 * n)
        field = mlcg_b200.GraphedForceField(model, make(frames[0].clone()))
        bnn.set_edge_capacity(model, None)
    wrong = torch.zeros((), dtype=torch.int64, device=DEV)
    for turn in range(300):
        k = turn % 3
        write(k)
        out = model(make(here)).out["SchNet"]
        pairs = [(out["energy"], out["forces"])] + ([] if field is None else [field(here)])
        for e, f in pairs:
            wrong += (e != want[k][0]).any() | (f != want[k][1]).any()
    assert int(wrong) == 0
    get_backend().check_pending()


@pytest.mark.parametrize("shift,table", [(0, False), (1, False), (2, False), (0, True), (3, True)])
@pytest.mark.parametrize("sizes", [[73], [60] * 30])
def test_weights_at_any_address(sizes, shift, table):
    """Small batches whose weights are parts of a larger buffer, on no 16-byte boundary: evaluations with forces, with a given list, in a fixed
    capacity, and steps.  Each is that of the same weights in buffers of their own, to the accuracy of the evaluation."""
    torch.manual_seed(3)
    cut = bnn.CosineCutoff(0.0, 8.0)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 33, trainable=False), cut, [64], embedding_size=5, num_interactions=2).to(DEV)
    model, gen, n = bnn.GradientsOut(net, "forces"), torch.Generator().manual_seed(1), sum(sizes)
    pos, types_ = torch.cat([random_walk_chain(k, gen, min_dist=3.0) for k in sizes]).to(DEV), (torch.arange(n) % 5).to(DEV)
    batch = torch.arange(len(sizes), device=DEV).repeat_interleave(torch.tensor(sizes, device=DEV))
    make = lambda: mlcg_b200.AtomicData(pos=pos.clone(), atom_types=types_, batch=batch, n_atoms=torch.tensor(sizes, device=DEV))  # noqa: E731

    def every():
        out = []
        model.eval()
        given = make()
        given.neighbor_list = net.neighbor_list(given, 8.0)
        E = given.neighbor_list["SchNet"]["index_mapping"].shape[1]
        for data, capacity in ((make(), None), (given, None), (make(), E + 2)):
            bnn.set_edge_capacity(model, capacity)
            o = model(data).out["SchNet"]
            out += [o["energy"].detach().clone(), o["forces"].detach().clone()]
        bnn.set_edge_capacity(model, None)
        model.train()
        net.zero_grad()
        o = model(make()).out["SchNet"]
        (o["forces"] ** 2).mean().backward()
        get_backend().check_pending()
        return out + [o["energy"].detach().clone(), o["forces"].detach().clone()] + [p.grad.clone() for p in net.parameters()]

    want = every()
    for name, p in net.named_parameters():
        k = shift if "embedding" not in name else (1 if table else 0)
        p.data = torch.cat([p.data.new_zeros(k), p.data.flatten()])[k:].view(p.shape)
    assert (net.embedding_layer.weight.data_ptr() % 16 != 0) == table
    for a, b in zip(every(), want):
        # (either side within 2e-5 of the largest entry, what steps hold against float64)
        assert float((a - b).abs().max()) <= 4e-5 * float(b.abs().max()) + 1e-9


@pytest.mark.parametrize("moved", ["forward", "backward"])
def test_a_step_whose_weights_change_place(moved):
    """Saved-tensor hooks that bring the weights back on other boundaries than the forward pass met: one pass by the chain of small batches, the
    other by the kernels of larger ones, over one workspace."""
    torch.manual_seed(3)
    cut = bnn.CosineCutoff(0.0, 8.0)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 33, trainable=False), cut, [64], embedding_size=5, num_interactions=3).to(DEV).train()
    model, gen = bnn.GradientsOut(net, "forces"), torch.Generator().manual_seed(1)
    pos, batch = torch.cat([random_walk_chain(60, gen, min_dist=3.0) for _ in range(4)]).to(DEV), torch.arange(4, device=DEV).repeat_interleave(60)
    weights = [p for name, p in net.named_parameters() if "embedding" not in name]

    def elsewhere(t, k):
        return torch.cat([t.new_zeros(k), t.detach().flatten()])[k:].view(t.shape)

    def step(pack, unpack):
        net.zero_grad()
        with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
            out = model(mlcg_b200.AtomicData(pos=pos, atom_types=torch.arange(240, device=DEV) % 5, batch=batch, n_atoms=torch.full((4,), 60, device=DEV))).out["SchNet"]
            ((out["forces"] ** 2).mean() + 0.01 * (out["energy"] ** 2).mean()).backward()
        assert type(out["forces"].grad_fn).__name__ == "SchNetForceMatchingBackward"
        return [p.grad.clone() for p in net.parameters()]

    want = step(lambda t: t, lambda t: t)
    if moved == "forward":
        for p in weights:
            p.data = elsewhere(p.data, 1)
    k, seen = int(moved == "backward"), []

    def back(t):
        if t.dtype == torch.float32 and any(t.shape == p.shape for p in weights):
            seen.append(t.shape)
            return elsewhere(t, k)
        return t

    got = step(lambda t: t, back)
    assert len(seen) >= len(weights)
    for a, b in zip(got, want):
        assert float((a - b).abs().max()) <= 4e-5 * float(b.abs().max()) + 1e-9      # (either side within 2e-5, as above)
    get_backend().check_pending()


@pytest.mark.parametrize("blocks", [1, 2])
def test_large_batches_with_nodes_of_every_degree(blocks):
    """Above the small batches' limit the last dot products are taken per pair: beads without neighbours, with one, and with several
    chunks of 32, the first upper neighbour anywhere in a chunk."""
    gen = torch.Generator().manual_seed(blocks)
    torch.manual_seed(2)
    upper, sizes = 6.0, [2200, 1, 2, 110, 150]
    cut = bnn.CosineCutoff(0.0, upper)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 32, trainable=False), cut, [128], hidden_channels=128, embedding_size=6, num_filters=128,
                             num_interactions=blocks)
    parts = [torch.rand(n, 3, generator=gen) * side for n, side in zip(sizes, (60.0, 1.0, 100.0, 9.0, 12.0))]
    parts[2] = torch.tensor([[0.0, 0.0, 0.0], [3.0, 0.0, 0.0]])
    pos = torch.cat(parts)
    types_, batch = torch.randint(0, 6, (sum(sizes),), generator=gen), torch.arange(len(sizes)).repeat_interleave(torch.tensor(sizes))
    e_x, f_x, _ = _oracle(net, "expnormal", upper, blocks, pos, types_, batch, len(sizes), torch.float64)
    net = net.to(DEV).eval()
    data = mlcg_b200.AtomicData(pos=pos.to(DEV), atom_types=types_.to(DEV), batch=batch.to(DEV), n_atoms=torch.tensor(sizes).to(DEV))
    degrees = net.neighbor_list(data, upper)["SchNet"]["index_mapping"][0].bincount(minlength=sum(sizes))
    assert int(degrees.min()) == 0 and int((degrees == 1).sum()) > 0 and int(degrees.max()) > 64
    out = bnn.GradientsOut(net, "forces").eval()(data).out["SchNet"]
    assert torch.allclose(out["energy"].cpu().double(), e_x, rtol=E_RTOL, atol=E_RTOL * float(e_x.abs().max()))
    # (dense clusters: forces of hundreds, to the same number of digits as elsewhere)
    assert float((out["forces"].cpu().double() - f_x).abs().max()) < F_ATOL * max(1.0, float(f_x.abs().max()) / 10)


@pytest.mark.parametrize("num_rbf,head,shift,too_large", [(20, 128, 0, None), (33, 64, 1, None), (64, 36, 2, None), (65, 4, 0, None), (128, 128, 3, None),
                                                          (50, 128, 0, "lin1"), (50, 128, 0, "filter2"), (50, 64, 0, "head")])
def test_weights_as_operand_tiles_of_large_batches(num_rbf, head, shift, too_large):
    """Above the small batches' limit the weights are made into operand tiles in front: of every width, at addresses of any alignment, and
    those beyond the range of a pair of fp16 are reported."""
    gen = torch.Generator().manual_seed(num_rbf)
    torch.manual_seed(3)
    upper, sizes = 8.0, [60] * 39 + [29]
    cut = bnn.CosineCutoff(0.0, upper)
    net = bnn.StandardSchNet(bnn.GaussianBasis(cut, num_rbf, trainable=False), cut, [head], hidden_channels=128, embedding_size=6, num_filters=128, num_interactions=2)
    pos = torch.cat([torch.rand(n, 3, generator=gen) * 14.0 for n in sizes])
    types_, batch = torch.randint(0, 6, (sum(sizes),), generator=gen), torch.arange(len(sizes)).repeat_interleave(torch.tensor(sizes))
    e_x, f_x, _ = _oracle(net, "gaussian", upper, 2, pos, types_, batch, len(sizes), torch.float64)
    net = net.to(DEV).eval()
    layers = dict(lin1=net.interaction_blocks[1].conv.lin1, filter2=[m for m in net.interaction_blocks[0].conv.filter_network.modules() if hasattr(m, "weight")][-1],
                  head=[m for m in net.output_network.modules() if hasattr(m, "weight")][0])
    for name, p in net.named_parameters():
        if "embedding" not in name:                    # (its rows are read in 16-byte pieces)
            p.data = torch.cat([p.data.new_zeros(shift), p.data.flatten()])[shift:].view(p.shape)
    if too_large:
        layers[too_large].weight.data[3, 1] = 600.0
    out = bnn.GradientsOut(net, "forces").eval()(mlcg_b200.AtomicData(pos=pos.to(DEV), atom_types=types_.to(DEV), batch=batch.to(DEV),
                                                                      n_atoms=torch.tensor(sizes).to(DEV))).out["SchNet"]
    if too_large:
        with pytest.raises(RuntimeError):
            get_backend().check_pending()
        return
    assert torch.allclose(out["energy"].cpu().double(), e_x, rtol=E_RTOL, atol=E_RTOL * float(e_x.abs().max()))
    assert float((out["forces"].cpu().double() - f_x).abs().max()) < F_ATOL * max(1.0, float(f_x.abs().max()) / 10)


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("basis,num_rbf,upper", [("expnormal", 128, 10.0), ("expnormal", 100, 15.0), ("gaussian", 128, 15.0), ("gaussian", 33, 30.0)])
def test_distances_on_both_sides_of_the_basis_that_is_zero(basis, num_rbf, upper, precision):
    """Pairs of two beads at distances from almost nothing to beyond the cutoff: quarters of the basis that are zero for a warp, for a tile,
    or for none, tiles of one kind and mixed ones, several tiles per block."""
    torch.manual_seed(4)
    cut = bnn.CosineCutoff(0.0, upper)
    kind = {"expnormal": bnn.ExpNormalBasis, "gaussian": bnn.GaussianBasis}[basis]
    net = bnn.StandardSchNet(kind(cut, num_rbf, trainable=False), cut, [128], hidden_channels=128, embedding_size=4, num_filters=128, num_interactions=1)
    pairs = 900
    gen = torch.Generator().manual_seed(5)
    d = torch.cat([torch.linspace(0.05, 1.02 * upper, pairs - 300), torch.full((150,), 0.9 * upper), torch.full((150,), 0.3)])
    d[300:450] = d[300:450][torch.randperm(150, generator=gen)]
    pos = torch.zeros(2 * pairs, 3)
    pos[1::2, 0] = d
    types_, batch = torch.randint(0, 4, (2 * pairs,), generator=gen), torch.arange(pairs).repeat_interleave(2)
    e_x, f_x, _ = _oracle(net, basis, upper, 1, pos, types_, batch, pairs, torch.float64)
    bnn.set_filter_precision(net.to(DEV).eval(), precision)
    out = bnn.GradientsOut(net, "forces").eval()(mlcg_b200.AtomicData(pos=pos.to(DEV), atom_types=types_.to(DEV), batch=batch.to(DEV),
                                                                      n_atoms=torch.full((pairs,), 2).to(DEV))).out["SchNet"]
    e, f = out["energy"].cpu().double(), out["forces"].cpu().double()
    if precision == "fp32":
        assert torch.allclose(e, e_x, rtol=E_RTOL, atol=E_RTOL * float(e_x.abs().max())) and float((f - f_x).abs().max()) < F_ATOL
    else:
        assert float((f - f_x).norm() / f_x.norm()) < 1e-2


@pytest.mark.parametrize("sizes,box,edges", [([1, 1, 1], 1.0, 0), ([4, 3], 3.0, 18), ([600, 1, 700], 3000.0, None), ([2048], 6000.0, None)])
def test_lists_without_room_for_an_edge(sizes, box, edges):
    """A fixed capacity of 0: beads alone get their energies, and every edge is reported.  Between the calls the workspaces hold lists of
    another batch, so that a link which reads them too early would read those."""
    import ctypes
    torch.manual_seed(0)
    cut = bnn.CosineCutoff(0.0, 6.0)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 32, trainable=False), cut, [128], embedding_size=5, num_interactions=2).eval().to(DEV)
    be, lib, n, gen = get_backend(), get_backend().lib, sum(sizes), torch.Generator().manual_seed(7)
    pos, types_ = (torch.rand(n, 3, generator=gen) * box).to(DEV), torch.randint(0, 5, (n,), generator=gen).to(DEV)
    n_atoms = torch.tensor(sizes, device=DEV)
    spec, conv_cut, (w, _keep), precision = net._whole_model_setup(pos)
    s, keep = be._spec(spec, torch.float32)
    size = lib.mlcgb_schnet_evaluate_workspace_bytes
    gb, wsb = size(n, len(sizes), -1, 0, ctypes.byref(w), 0), size(n, len(sizes), 0, spec.num_rbf, ctypes.byref(w), 0)
    status, per_type = be._sticky_status(torch.device(DEV)), None
    alone = bnn.GradientsOut(net, "forces").eval()(mlcg_b200.AtomicData(pos=torch.arange(5, device=DEV)[:, None] * torch.full((1, 3), 50.0, device=DEV), atom_types=torch.arange(5, device=DEV),
                                                                      batch=torch.arange(5, device=DEV), n_atoms=torch.ones(5, dtype=torch.int64, device=DEV)))
    per_type = alone.out["SchNet"]["energy"]
    want = torch.zeros(len(sizes), device=DEV).index_add_(0, torch.repeat_interleave(torch.arange(len(sizes), device=DEV), n_atoms), per_type[types_])
    for fill in (0, 1, 0x7f):
        graph_ws, ws = (torch.full((b,), fill, dtype=torch.uint8, device=DEV) for b in (gb, wsb))
        energy, grad = torch.empty(len(sizes), device=DEV), torch.empty(n, 3, device=DEV)
        code = lib.mlcgb_schnet_evaluate_fixed(pos.data_ptr(), types_.data_ptr(), n_atoms.data_ptr(), None, n, len(sizes), 6.0, 1000, ctypes.byref(s), conv_cut[0],
                                               conv_cut[1], conv_cut[2], ctypes.byref(w), precision, 1, 0, None, graph_ws.data_ptr(), gb, ws.data_ptr(), wsb,
                                               energy.data_ptr(), grad.data_ptr(), status.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert code == 0 and int(status[0]) == (32 if edges else 0)
        status.zero_()
        assert torch.allclose(energy, want, rtol=1e-5, atol=1e-5 * float(want.abs().max())) and not grad.any()


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("num_rbf", [128, 50, 33])
@pytest.mark.parametrize("copies", [3, 600])
def test_a_weight_that_is_not_a_number_reaches_the_results(copies, num_rbf, precision):
    """Also where it stands in a column of the filter network's first layer that the basis does not reach: energies and forces are no
    numbers either, in batches of both routes."""
    torch.manual_seed(4)
    cut = bnn.CosineCutoff(0.0, 10.0)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, num_rbf, trainable=False), cut, [128], hidden_channels=128, embedding_size=4, num_filters=128, num_interactions=2)
    model = bnn.GradientsOut(bnn.set_filter_precision(net.to(DEV).eval(), precision), "forces").eval()
    pos = random_walk_chain(5, torch.Generator().manual_seed(1), min_dist=3.8).repeat(copies, 1).to(DEV)
    batch = torch.arange(copies, device=DEV).repeat_interleave(5)
    data = lambda: mlcg_b200.AtomicData(pos=pos.clone(), atom_types=torch.zeros(5 * copies, dtype=torch.int64, device=DEV), batch=batch,  # noqa: E731
                                        n_atoms=torch.full((copies,), 5, device=DEV))
    want = model(data()).out["SchNet"]
    assert bool(want["energy"].isfinite().all() and want["forces"].isfinite().all())
    layers = net.interaction_blocks[1].conv.filter_network.layers
    for weight, places in ((layers[0].weight, ((0, 0), (17, num_rbf - 1), (127, num_rbf // 2))), (layers[0].bias, ((5,),)), (layers[2].weight, ((3, 64),))):
        for at in places:
            before = weight.data[at].clone()
            weight.data[at] = float("nan")
            out = model(data()).out["SchNet"]
            assert bool(out["energy"].isnan().all()) and bool(out["forces"].isnan().all()), (tuple(weight.shape), at)
            weight.data[at] = before
    again = model(data()).out["SchNet"]
    assert torch.equal(again["energy"], want["energy"]) and torch.equal(again["forces"], want["forces"])


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("blocks", [1, 2, 3])
def test_few_tiles_of_pairs_in_two_ctas_each(blocks, precision):
    """With a tile of pairs for every second SM or less, values and derivatives of a tile go to two CTAs: 31 beads make 465 pairs (four tiles),
    twenty times as many 73 tiles, forty times 146.  The same structure has the same numbers in each, but for the order in which the parts
    of a bead's 30 edges are added up, which goes by the size of the batch: 30 roundings of the largest partial sum, taken as 32 times
    the largest force."""
    torch.manual_seed(blocks)
    cut = bnn.CosineCutoff(0.0, 60.0)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 64, trainable=False), cut, [128], hidden_channels=128, embedding_size=4, num_filters=128, num_interactions=blocks)
    model = bnn.GradientsOut(bnn.set_filter_precision(net.to(DEV).eval(), precision), "forces").eval()
    one, types_ = torch.rand(31, 3, generator=torch.Generator().manual_seed(7)).mul(14.0).to(DEV), (torch.arange(31) % 4).to(DEV)
    got = []
    for copies in (1, 20, 40):
        batch, sizes = torch.arange(copies, device=DEV).repeat_interleave(31), torch.full((copies,), 31, device=DEV)
        out = model(mlcg_b200.AtomicData(pos=one.repeat(copies, 1), atom_types=types_.repeat(copies), batch=batch, n_atoms=sizes)).out["SchNet"]
        forces = out["forces"].view(copies, 31, 3)
        assert torch.equal(forces, forces[:1].expand_as(forces)) and torch.equal(out["energy"], out["energy"][:1].expand_as(out["energy"]))
        got.append((out["energy"][0], forces[0]))
    for energy, forces in got[1:]:
        assert float((forces - got[0][1]).abs().max()) <= 30 * 2.0 ** -24 * 32 * float(got[0][1].abs().max())
        assert torch.allclose(energy, got[0][0], rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("blocks", [1, 2, 3])
def test_filter_rows_of_two_ctas_are_those_of_one(blocks):
    """The rows themselves: 40 copies of the 31 beads have 146 tiles of pairs, one CTA for each, and the first copy's rows and derivatives are, bit by bit,
    those of the copy alone, in two CTAs a tile.  Read from the workspace of a step's forward pass (its arrays lie on 256-byte boundaries:
    positions, edges, edges, pairs, beads, output network, one per block, then the rows of all blocks and their derivatives)."""
    from mlcg_b200.autograd import plan_of
    torch.manual_seed(blocks)
    cut, head = bnn.CosineCutoff(0.0, 60.0), 64
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 64, trainable=False), cut, [head], embedding_size=4, num_interactions=blocks).to(DEV).train()
    one, types_ = torch.rand(31, 3, generator=torch.Generator().manual_seed(7)).mul(14.0).to(DEV), (torch.arange(31) % 4).to(DEV)
    rows = []
    for copies in (1, 40):
        N, P = 31 * copies, 465 * copies
        data = mlcg_b200.AtomicData(pos=one.repeat(copies, 1), atom_types=types_.repeat(copies), batch=torch.arange(copies, device=DEV).repeat_interleave(31),
                                    n_atoms=torch.full((copies,), 31, device=DEV))
        nl = net.neighbor_list(data, 60.0)["SchNet"]
        plan = plan_of(nl["index_mapping"], N)
        assert plan.E == 2 * P and N <= 2368
        state = get_backend().schnet_train_forward(data.pos, data.atom_types, nl["_mlcgb_ptr"], plan, *net._whole_model_setup(data.pos, training=True)[:3])[2]
        ws = state.tensors[state.places[state.NAMES.index("forward_ws")][0]].view(torch.float32)
        at, stride = sum((k + 63) // 64 * 64 for k in (3 * N, 2 * P, 2 * P, P, N, N * head, blocks)), (P + 127) // 128 * 128 * 128
        values, derivatives = (ws[at + k * blocks * stride: at + (k + 1) * blocks * stride].view(blocks, -1, 128)[:, :465] for k in (0, 1))
        first = plan.half_selection()[:465]
        rows.append((values.clone(), derivatives.clone(), plan.row0[first].clone(), plan.row1[first].clone()))
    assert float(rows[0][0].abs().max()) > 0 and float(rows[0][1].abs().max()) > 0
    assert all(torch.equal(a, b) for a, b in zip(*rows))
    get_backend().check_pending()


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_evaluations_repeat_bit_by_bit(precision):
    """The node layers' parts of tiles are copied into places that have just been read: a copy that overtakes the reads shows up as rows of
    the wrong matrix, once in some hundred evaluations of this batch (24 tiles of beads, two blocks)."""
    torch.manual_seed(4)
    cut = bnn.CosineCutoff(0.0, 10.0)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 128, trainable=False), cut, [128], hidden_channels=128, embedding_size=4, num_filters=128, num_interactions=2)
    model = bnn.GradientsOut(bnn.set_filter_precision(net.to(DEV).eval(), precision), "forces").eval()
    pos, batch = random_walk_chain(5, torch.Generator().manual_seed(1), min_dist=3.8).repeat(600, 1).to(DEV), torch.arange(600, device=DEV).repeat_interleave(5)
    types_, sizes = torch.zeros(3000, dtype=torch.int64, device=DEV), torch.full((600,), 5, device=DEV)
    step = lambda: model(mlcg_b200.AtomicData(pos=pos, atom_types=types_, batch=batch, n_atoms=sizes)).out["SchNet"]  # noqa: E731
    want, differs = step(), torch.zeros((), dtype=torch.int64, device=DEV)
    for _ in range(2000):
        got = step()
        differs += (got["forces"] != want["forces"]).any() | (got["energy"] != want["energy"]).any()
    assert int(differs) == 0


@pytest.mark.parametrize("sizes", [[2049], [1500, 1400], [100] * 30])
def test_room_of_large_batches(sizes):
    """Above 2048 beads the workspace goes by the call before: one that is too small, exact or larger gives the evaluation of a given list."""
    torch.manual_seed(0)
    cut = bnn.CosineCutoff(0.0, 6.0)
    net = bnn.StandardSchNet(bnn.ExpNormalBasis(cut, 32, trainable=False), cut, [128], embedding_size=5, num_interactions=2).eval().to(DEV)
    model, n, gen = bnn.GradientsOut(net, "forces").eval(), sum(sizes), torch.Generator().manual_seed(1)
    pos, types_ = (torch.rand(n, 3, generator=gen) * 2.5 * max(sizes) ** (1 / 3)).to(DEV), torch.randint(0, 5, (n,), generator=gen).to(DEV)
    make = lambda: mlcg_b200.AtomicData(pos=pos.clone(), atom_types=types_, batch=torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes)).to(DEV),  # noqa: E731
                                        n_atoms=torch.tensor(sizes, device=DEV))
    given = make()
    given.neighbor_list = net.neighbor_list(given, 6.0)
    E = given.neighbor_list["SchNet"]["index_mapping"].shape[1]
    want = model(given).out["SchNet"]
    for guess in (0.0, (E - 2) / n / 1.04, E / n, 3 * E / n):
        net.__dict__["_mlcgb_edges_per_bead_large"] = guess
        got = model(make()).out["SchNet"]
        assert torch.equal(got["energy"], want["energy"]) and torch.equal(got["forces"], want["forces"]), guess
        assert net.__dict__["_mlcgb_edges_per_bead_large"] == E / n
