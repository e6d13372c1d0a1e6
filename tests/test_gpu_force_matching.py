"""The one-call force-matching step (values, forces, weight gradients) against a float64 evaluation of the same float32 weights."""
import copy
import io

import pytest
import torch

import mlcg_b200
from mlcg_b200 import nn as bnn
from oracle import radius_ref, schnet_ref

from helpers import random_walk_chain

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _setup(kind, R, upper, L, sizes, head, seed):
    gen = torch.Generator().manual_seed(seed)
    torch.manual_seed(seed)
    cut = bnn.CosineCutoff(0.0, upper)
    basis = bnn.GaussianBasis if kind == "gaussian" else bnn.ExpNormalBasis
    net = bnn.StandardSchNet(basis(cut, R, trainable=False), cut, [head], hidden_channels=128, embedding_size=7, num_filters=128, num_interactions=L)
    with torch.no_grad():
        for n, p in net.named_parameters():
            if n.endswith("bias"):
                p.normal_(0.0, 0.1)
    pos = torch.cat([random_walk_chain(n, gen, jitter=0.2) for n in sizes])
    types_ = torch.randint(0, 7, (len(pos),), generator=gen)
    batch = torch.arange(len(sizes)).repeat_interleave(torch.tensor(sizes))
    target = torch.randn(len(pos), 3, generator=gen)
    return net, pos, types_, batch, target


def _reference(net, kind, upper, L, pos, types_, batch, B, loss_of):
    cut = {"cutoff": "cosine", "lower": 0.0, "upper": upper}
    spec = {"kind": kind, "rbf_cutoff": cut, "cutoff": cut, "activation": "tanh", "num_interactions": L}
    names = {n for n, _ in net.named_parameters()}
    sd = {k: (v.detach().cpu().double().requires_grad_(k in names) if v.is_floating_point() else v.cpu()) for k, v in net.state_dict().items()}
    ei = torch.from_numpy(radius_ref.radius_graph_c(pos.numpy(), radius_ref.batch_to_ptr(batch.numpy(), B), upper, 1000, False, "cluster"))
    p = pos.double().requires_grad_(True)
    e = schnet_ref.schnet_energy(sd, spec, p, types_, batch, ei, B)
    f = -torch.autograd.grad(e.sum(), p, create_graph=True)[0]
    loss = loss_of(e, f)
    grads = torch.autograd.grad(loss, [sd[n] for n in sorted(names)], allow_unused=True)
    return e.detach(), f.detach(), loss.detach(), dict(zip(sorted(names), grads))


@pytest.mark.parametrize("kind,R,upper,L,sizes,head,energies", [
    ("expnormal", 128, 10.0, 3, [73] * 6, 128, False),       # several tiles of pairs and nodes
    ("gaussian", 50, 30.0, 2, [10] * 13, 128, True),         # a basis narrower than half a tile, energies in the loss
    ("gaussian", 65, 9.0, 1, [5, 40, 23], 64, True),         # one block (no tangent into it), a narrow output network
    ("expnormal", 20, 12.0, 2, [2], 128, False),             # one pair
    ("expnormal", 64, 8.0, 3, [129, 1, 17], 32, True),       # a bead without neighbours
    ("expnormal", 100, 11.0, 2, [300], 128, False),
    ("gaussian", 50, 8.0, 2, [74] * 32 + [9], 96, True),     # more beads than the small route takes
])
def test_step_against_float64(kind, R, upper, L, sizes, head, energies):
    net, pos, types_, batch, target = _setup(kind, R, upper, L, sizes, head, 3)
    B = len(sizes)
    loss_of = lambda e, f: ((f - target.to(f)) ** 2).mean() + (0.01 * (e ** 2).mean() if energies else 0.0)  # noqa: E731
    e_x, f_x, loss_x, g_x = _reference(net, kind, upper, L, pos, types_, batch, B, loss_of)
    net = net.to(DEV).train()
    assert net._whole_model_setup(pos.to(DEV), training=True) is not None
    data = lambda: mlcg_b200.AtomicData(pos=pos.to(DEV), atom_types=types_.to(DEV), batch=batch.to(DEV), n_atoms=torch.tensor(sizes).to(DEV))  # noqa: E731
    out = bnn.GradientsOut(net, "forces").train()(data()).out["SchNet"]
    assert type(out["forces"].grad_fn).__name__ == "SchNetForceMatchingBackward"
    loss = loss_of(out["energy"], out["forces"])
    loss.backward()
    assert float((out["energy"].detach().cpu().double() - e_x).abs().max()) < 1e-5 * float(e_x.abs().max() + 1e-3)
    assert float((out["forces"].detach().cpu().double() - f_x).abs().max()) < 1e-4
    assert abs(float(loss.detach()) - float(loss_x)) < 1e-5 * float(loss_x)
    for n, p in net.named_parameters():
        g = g_x[n]
        if g is None:
            continue
        assert float((p.grad.cpu().double() - g).abs().max()) <= 2e-5 * float(g.abs().max()) + 1e-9, n


@pytest.mark.parametrize("beads", [74, 75, 148, 149, 222, 223, 592, 593, 888, 889, 1184, 1185, 1776, 1777, 2368])
def test_tiles_of_every_height(beads):
    """Small batches run in tiles of 1 to 8 rows by their number of beads: both sides of every line, forward and backward."""
    sizes = [37] * (beads // 37) + [beads % 37] * (beads % 37 > 0)
    test_step_against_float64("expnormal", 20, 7.0, 2, sizes, 128, True)


@pytest.mark.parametrize("beads", [73, 200])
def test_more_edges_than_the_tiles_of_beads_have_threads(beads):
    """Above 64 edges a bead the first launch of a small step has CTAs of edges alone, which bring no weights: every pair of one chain."""
    assert beads * (beads - 1) > 512 * ((beads + 7) // 8)
    test_step_against_float64("gaussian", 64, {73: 40.0, 200: 95.0}[beads], 2, [beads], 128, True)


@pytest.mark.parametrize("copies,head", [(3789, 128), (7579, 96)])
def test_linked_layers_over_several_tiles_each(copies, head):
    """More tiles of 128 beads than the chip has SMs: 18945 beads, the last tile one row high, and two tiles for each and seven beads.  The same
    structure over and over has the same energies and forces in every copy and every call, those of one copy alone, and the gradients of
    one copy alone, in steps and in evaluations."""
    net, pos, types_, _, target = _setup("expnormal", 32, 9.0, 3, [5], head, 11)
    net = net.to(DEV)
    model, n = bnn.GradientsOut(net, "forces"), 5

    def data(k):
        return mlcg_b200.AtomicData(pos=pos.repeat(k, 1).to(DEV), atom_types=types_.repeat(k).to(DEV), batch=torch.arange(k, device=DEV).repeat_interleave(n),
                                    n_atoms=torch.full((k,), n, device=DEV))

    def step(k):
        model.train()
        net.zero_grad()
        out = model(data(k)).out["SchNet"]
        assert type(out["forces"].grad_fn).__name__ == "SchNetForceMatchingBackward"
        (((out["forces"] - target.repeat(k, 1).to(DEV)) ** 2).sum() / k + 0.01 * (out["energy"] ** 2).sum() / k).backward()
        return out["energy"].detach().clone(), out["forces"].detach().clone(), [p.grad.clone() for p in net.parameters()]

    def evaluation(k):
        out = model.eval()(data(k)).out["SchNet"]
        return out["energy"].clone(), out["forces"].clone()

    for call, times in ((evaluation, 40), (step, 10)):
        one, many = call(1), call(copies)
        assert torch.equal(many[0], many[0][:1].expand(copies)) and torch.equal(many[1].view(copies, n, 3), many[1][:n].expand(copies, n, 3))
        # (either within 1e-5 and 1e-4 of float64, and gradients within 2e-5 of the largest, as above)
        assert torch.allclose(many[0][:1], one[0], rtol=2e-5, atol=2e-5) and float((many[1][:n] - one[1]).abs().max()) < 2e-4
        for a, b in zip(*(x[2] if len(x) > 2 else [] for x in (many, one))):
            assert float((a - b).abs().max()) <= 4e-5 * float(b.abs().max()) + 1e-9
        for _ in range(times):
            got = call(copies)
            assert torch.equal(got[0], many[0]) and torch.equal(got[1], many[1])
            assert all(torch.equal(a, b) for a, b in zip(*(x[2] if len(x) > 2 else [] for x in (got, many))))


def test_higher_derivatives_and_position_gradients_take_the_composable_operators():
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, [12, 9], 128, 5)
    net = net.to(DEV)
    m = bnn.GradientsOut(net, "forces").train()
    mk = lambda p: mlcg_b200.AtomicData(pos=p, atom_types=types_.to(DEV), batch=batch.to(DEV), n_atoms=torch.tensor([12, 9]).to(DEV))  # noqa: E731
    params = [p for n, p in net.named_parameters()]
    first = {}
    for fused in (True, False):
        p = pos.to(DEV).requires_grad_(not fused)
        loss = ((m(mk(p)).out["SchNet"]["forces"] - target.to(DEV)) ** 2).mean()
        g = torch.autograd.grad(loss, params, create_graph=True)
        norm = sum((x ** 2).sum() for x in g)
        first[fused] = torch.autograd.grad(norm, params[:6])
    for a, b in zip(first[True], first[False]):
        assert torch.allclose(a, b, rtol=1e-3, atol=1e-4 * float(b.abs().max()))
    p = pos.to(DEV).requires_grad_(True)
    ((m(mk(p)).out["SchNet"]["forces"] - target.to(DEV)) ** 2).mean().backward()
    assert p.grad is not None and bool(torch.isfinite(p.grad).all()) and float(p.grad.abs().max()) > 0


def test_a_step_leaves_nothing_behind():
    """Device memory is the same after every step: the graph of a step is freed with its outputs."""
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, [40] * 8, 128, 7)
    m = bnn.GradientsOut(net.to(DEV), "forces").train()
    used = []
    for _ in range(4):
        data = mlcg_b200.AtomicData(pos=pos.to(DEV), atom_types=types_.to(DEV), batch=batch.to(DEV), n_atoms=torch.full((8,), 40).to(DEV))
        ((m(data).out["SchNet"]["forces"] - target.to(DEV)) ** 2).mean().backward()
        net.zero_grad(set_to_none=True)
        del data
        used.append(torch.cuda.memory_allocated())
    assert used[1] == used[2] == used[3]


def _data(pos, types_, sizes, **more):
    n = torch.tensor(sizes)
    return mlcg_b200.AtomicData(pos=pos.to(DEV, copy=True), atom_types=types_.to(DEV, copy=True), batch=torch.arange(len(n)).repeat_interleave(n).to(DEV),
                                n_atoms=n.to(DEV), **more)


def _fused(value):
    return type(value.grad_fn).__name__ == "SchNetForceMatchingBackward"


def _grads(net):
    return {n: p.grad.clone() for n, p in net.named_parameters() if p.grad is not None}


def _step(m, data, target):
    m.zero_grad(set_to_none=True)
    out = m(data).out["SchNet"]
    ((out["forces"] - target.to(DEV)) ** 2).mean().backward()
    return out


def _close(a, b, rtol=1e-4):
    assert a.keys() == b.keys()
    for n in a:
        assert float((a[n] - b[n]).abs().max()) <= rtol * float(b[n].abs().max()) + 1e-9, n


@pytest.mark.parametrize("given_list", [False, True])
def test_the_backward_frees_what_the_forward_kept(given_list):
    """The state of a forward pass belongs to its autograd node: gone after the backward although the outputs live on, and seen by
    saved-tensor hooks, which may bring it back at another address."""
    sizes = [40] * 8
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 7)
    m = bnn.GradientsOut(net.to(DEV), "forces").train()
    more = {}
    if given_list:
        more["neighbor_list"] = net.neighbor_list(_data(pos, types_, sizes), 9.0)
    kept = 4 * 2 * 512 * 2000          # W, W', h and z of two blocks and at least 2000 pairs
    _step(m, _data(pos, types_, sizes, **more), target)
    plain = _grads(net)
    before = torch.cuda.memory_allocated()
    out = _step(m, _data(pos, types_, sizes, **more), target)
    assert _fused(out["forces"])
    assert torch.cuda.memory_allocated() - before < kept // 8
    seen = []

    def pack(t):
        seen.append(t.numel() * t.element_size())
        return t.cpu()

    m.zero_grad(set_to_none=True)
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.to(DEV)):
        out = m(_data(pos, types_, sizes, **more)).out["SchNet"]
        loss = ((out["forces"] - target.to(DEV)) ** 2).mean()
    assert sum(seen) > kept
    junk = [torch.full((sum(seen) // 4,), float("nan"), device=DEV) for _ in range(2)]     # (where the forward's buffers were)
    loss.backward()
    _close(_grads(net), plain, 1e-6)
    del junk


def test_inputs_overwritten_before_the_backward():
    """The next batch copied over the positions leaves the gradients alone; bead types that changed are an error, as anywhere in torch."""
    sizes = [23, 40, 9]
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 8)
    m = bnn.GradientsOut(net.to(DEV), "forces").train()
    _step(m, _data(pos, types_, sizes), target)
    expected = _grads(net)
    for given_list in (False, True):
        data = _data(pos, types_, sizes)
        if given_list:
            data.neighbor_list = net.neighbor_list(data, 9.0)
        mine = data.pos
        m.zero_grad(set_to_none=True)
        out = m(data).out["SchNet"]
        assert _fused(out["forces"])
        with torch.no_grad():
            mine.copy_(mine.flip(0) * 1.5)
        data.n_atoms.zero_()
        ((out["forces"] - target.to(DEV)) ** 2).mean().backward()
        _close(_grads(net), expected, 1e-6)
    data = _data(pos, types_, sizes)
    out = m(data).out["SchNet"]
    data.atom_types.zero_()
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out["forces"].sum().backward()


@pytest.mark.parametrize("training", [True, False])
def test_a_layer_replaced_after_a_call(training):
    sizes = [23, 40]
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 15)
    m = bnn.GradientsOut(net.to(DEV), "forces").train(training)
    before = m(_data(pos, types_, sizes)).out["SchNet"]["forces"].detach()
    for path, layer in (("interaction_blocks.0.conv.lin1", torch.nn.Linear(128, 128, bias=False)),
                        ("interaction_blocks.1.conv.filter_network.layers.0", torch.nn.Linear(32, 128)), ("output_network.layers.0", torch.nn.Linear(128, 128)),
                        ("interaction_blocks.0.activation", torch.nn.SiLU())):
        parent, _, name = path.rpartition(".")
        setattr(net.get_submodule(parent), name, layer.to(DEV))
        got = m(_data(pos, types_, sizes)).out["SchNet"]["forces"].detach()
        net2, *_ = _setup("expnormal", 32, 9.0, 2, sizes, 128, 15)
        net2.interaction_blocks[0].activation = copy.deepcopy(net.interaction_blocks[0].activation)
        net2.load_state_dict(net.state_dict())
        fresh = bnn.GradientsOut(net2.to(DEV), "forces").train(training)(_data(pos, types_, sizes)).out["SchNet"]["forces"].detach()
        scale = float(fresh.abs().max())
        assert torch.allclose(got, fresh, rtol=1e-4, atol=1e-4 * scale) and float((got - before).abs().max()) > 1e-3 * scale, path
        before = got


@pytest.mark.parametrize("where", ["", "interaction_blocks.0", "interaction_blocks.1.conv", "embedding_layer", "output_network"])
def test_hooks_run_in_training(where):
    sizes = [23, 40]
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 9)
    net = net.to(DEV)
    m = bnn.GradientsOut(net, "forces").train()
    _step(m, _data(pos, types_, sizes), target)
    expected, calls = _grads(net), []
    handles = [net.get_submodule(where).register_forward_hook(lambda *a: calls.append("after")),
               net.get_submodule(where).register_forward_pre_hook(lambda *a: calls.append("before"))]
    _step(m, _data(pos, types_, sizes), target)
    assert calls == ["before", "after"]
    _close(_grads(net), expected)
    for h in handles:
        h.remove()
    assert _fused(_step(m, _data(pos, types_, sizes), target)["forces"])


@pytest.mark.parametrize("training", [True, False])
def test_a_forward_of_ones_own_runs(training):
    sizes = [23, 40]
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 9)

    class Shifted(bnn.StandardSchNet):
        def forward(self, data):
            data = super().forward(data)
            data.out[self.name]["energy"] = 2.0 * data.out[self.name]["energy"]
            return data

    m = bnn.GradientsOut(net.to(DEV), "forces").train(training)
    once = m(_data(pos, types_, sizes)).out["SchNet"]["energy"]
    net.__class__ = Shifted
    assert torch.allclose(m(_data(pos, types_, sizes)).out["SchNet"]["energy"], 2.0 * once, rtol=1e-5)


@pytest.mark.parametrize("option", [dict(padding_idx=2), dict(scale_grad_by_freq=True), dict(sparse=True), dict(max_norm=0.5)])
def test_options_of_the_embedding(option):
    sizes = [23, 40]
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 10)
    net = net.to(DEV)
    weight = net.embedding_layer.weight.detach().clone()
    grads = []
    for asked in (False, True):            # the composable operators, then what the model takes by itself
        net.embedding_layer = torch.nn.Embedding(7, 128, _weight=weight.clone(), **option)
        m = bnn.GradientsOut(net, "forces").train()
        data = _data(pos, types_, sizes)
        data.pos.requires_grad_(not asked)
        _step(m, data, target)
        grads.append({n: p.grad.to_dense().clone() for n, p in net.named_parameters()} | {"table": net.embedding_layer.weight.detach().clone()})
    _close(grads[1], grads[0])


@pytest.mark.parametrize("create_graph", [False, True])
def test_parameters_handed_in_for_a_call(create_graph):
    """``torch.func.functional_call`` with aliases of the weights, and with other values than the module's."""
    sizes = [23, 40]
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 11)
    m = bnn.GradientsOut(net.to(DEV), "forces").train()
    _step(m, _data(pos, types_, sizes), target)
    own = {n: p.grad.clone() for n, p in m.named_parameters() if p.grad is not None}
    m.zero_grad(set_to_none=True)
    for scale in (1.0, 1.1):
        given = {n: (p.detach() if scale == 1.0 else p.detach() * scale).requires_grad_() for n, p in m.named_parameters()}
        out = torch.func.functional_call(m, given, (_data(pos, types_, sizes),)).out["SchNet"]
        loss = ((out["forces"] - target.to(DEV)) ** 2).mean()
        got = torch.autograd.grad(loss, list(given.values()), create_graph=create_graph, allow_unused=True)
        got = {n: g.detach() for n, g in zip(given, got) if g is not None}
        if scale != 1.0:
            with torch.no_grad():
                for p in m.parameters():
                    p.mul_(scale)
            _step(m, _data(pos, types_, sizes), target)
            own = {n: p.grad.clone() for n, p in m.named_parameters() if p.grad is not None}
        assert set(own) <= set(got) | {"model.output_network.layers.2.bias"}
        _close({n: got[n] for n in own}, own)


def test_second_derivatives_of_a_shared_layer():
    """A filter network that two blocks share enters the step twice: its gradient is one sum, differentiable or not."""
    sizes = [23, 40]
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 16)
    net.interaction_blocks[1].conv.filter_network = net.interaction_blocks[0].conv.filter_network
    m = bnn.GradientsOut(net.to(DEV), "forces").train()
    _step(m, _data(pos, types_, sizes), target)
    expected = _grads(net)
    names = list(expected)
    for create_graph in (False, True):
        loss = ((m(_data(pos, types_, sizes)).out["SchNet"]["forces"] - target.to(DEV)) ** 2).mean()
        got = torch.autograd.grad(loss, [dict(net.named_parameters())[n] for n in names], create_graph=create_graph)
        _close(dict(zip(names, (g.detach() for g in got))), expected)


def test_a_basis_unfrozen_later_is_trained():
    sizes = [23, 40]
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 12)
    basis = bnn.ExpNormalBasis(net.rbf_layer.cutoff, 32, trainable=True).requires_grad_(False)
    net.rbf_layer = basis
    m = bnn.GradientsOut(net.to(DEV), "forces").train()
    assert _fused(_step(m, _data(pos, types_, sizes), target)["forces"]) and basis.means.grad is None
    basis.requires_grad_(True)
    _step(m, _data(pos, types_, sizes), target)
    assert basis.means.grad is not None and float(basis.means.grad.abs().max()) > 0
    basis.requires_grad_(False)
    assert _fused(_step(m, _data(pos, types_, sizes), target)["forces"])


class _Doubled(torch.nn.Module):
    def forward(self, w):
        return 2.0 * w


@pytest.mark.parametrize("ran_before", [False, True])
@pytest.mark.parametrize("layer", ["interaction_blocks.0.conv.lin1", "interaction_blocks.1.conv.filter_network.layers.2", "output_network.layers.0"])
def test_parametrized_weights(layer, ran_before):
    sizes = [23, 40]
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 14)
    net = net.to(DEV)
    m = bnn.GradientsOut(net, "forces").train()
    doubled = copy.deepcopy(net)
    with torch.no_grad():
        doubled.get_submodule(layer).weight.mul_(2.0)
    md = bnn.GradientsOut(doubled, "forces").train()
    expected = _step(md, _data(pos, types_, sizes), target)["forces"].detach()
    if ran_before:
        _step(m, _data(pos, types_, sizes), target)
    torch.nn.utils.parametrize.register_parametrization(net.get_submodule(layer), "weight", _Doubled())
    got = _step(m, _data(pos, types_, sizes), target)["forces"].detach()
    assert torch.allclose(got, expected, rtol=1e-4, atol=1e-4 * float(expected.abs().max()))
    w = net.get_submodule(layer).parametrizations.weight.original.grad
    assert torch.allclose(w, 2.0 * doubled.get_submodule(layer).weight.grad, rtol=1e-3, atol=1e-4 * float(w.abs().max()))
    for mode, ref in ((m.eval(), md.eval()),):
        assert torch.allclose(mode(_data(pos, types_, sizes)).out["SchNet"]["forces"], ref(_data(pos, types_, sizes)).out["SchNet"]["forces"],
                              rtol=1e-4, atol=1e-4 * float(expected.abs().max()))


def test_a_model_that_has_run_can_be_copied_and_saved():
    sizes = [23, 40]
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 13)
    m = bnn.GradientsOut(net.to(DEV), "forces").train()
    _step(m, _data(pos, types_, sizes), target)
    expected = _grads(net)
    m.eval()(_data(pos, types_, sizes))
    file = io.BytesIO()
    torch.save(m, file)
    file.seek(0)
    for other in (copy.deepcopy(m), torch.load(file, weights_only=False)):
        _step(other.train(), _data(pos, types_, sizes), target)
        _close(_grads(other.model), expected, 1e-6)


@pytest.mark.parametrize("training", [True, False])
def test_a_weight_turned_in_place_after_a_call(training):
    sizes = [23, 40]
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 17)
    net = net.to(DEV)
    m = bnn.GradientsOut(net, "forces").train(training)
    m(_data(pos, types_, sizes))
    w = net.interaction_blocks[1].conv.lin1.weight
    w.data = w.data.t()                            # same storage, other strides
    got = m(_data(pos, types_, sizes)).out["SchNet"]["forces"].detach()
    w.data = w.data.contiguous()
    expected = m(_data(pos, types_, sizes)).out["SchNet"]["forces"].detach()
    assert torch.allclose(got, expected, rtol=1e-4, atol=1e-4 * float(expected.abs().max()))


@pytest.mark.parametrize("training", [True, False])
def test_inputs_a_kernel_could_not_read_are_refused(training):
    """Bead types on the host, or fewer of them than beads, end in an error on the host."""
    sizes = [23, 40]
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 18)
    m = bnn.GradientsOut(net.to(DEV), "forces").train(training)
    for wrong in (types_, types_.to(DEV)[:-1]):
        for given_list in (False, True):
            data = _data(pos, types_, sizes)
            if given_list:
                data.neighbor_list = net.neighbor_list(data, 9.0)
            data.atom_types = wrong
            with pytest.raises((RuntimeError, ValueError)):
                m(data)


def test_a_checkpointed_step():
    """What a pass saves has the sizes of its edges, not of the guess before it: a checkpoint's second forward saves the same."""
    from torch.utils.checkpoint import checkpoint
    net, *_ = _setup("expnormal", 32, 9.0, 2, [40], 128, 19)
    m = bnn.GradientsOut(net.to(DEV), "forces").train()
    for sizes in ([40] * 4, [23, 40, 9], [73] * 3, [300]):
        _, pos, types_, _, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 20)
        m.zero_grad(set_to_none=True)
        forces = checkpoint(lambda p: m(_data(p, types_, sizes)).out["SchNet"]["forces"], pos.to(DEV), use_reentrant=False)
        ((forces - target.to(DEV)) ** 2).mean().backward()
        got = _grads(net)
        loss = ((m(_data(pos, types_, sizes)).out["SchNet"]["forces"] - target.to(DEV)) ** 2).mean()
        m.zero_grad(set_to_none=True)
        loss.backward(retain_graph=True)
        _close(got, _grads(net), 1e-6)
        m.zero_grad(set_to_none=True)
        loss.backward()                            # (a second backward over the same state)
        _close(_grads(net), got, 1e-6)


@pytest.mark.parametrize("training", [True, False])
def test_a_part_of_the_model_in_the_other_mode(training):
    """A block switched to the other mode after a call: its layers act as they do in a model that has had it so from the start."""
    sizes = [23, 40]
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 21)
    m = bnn.GradientsOut(net.to(DEV), "forces").train(training)
    other = copy.deepcopy(m)
    m(_data(pos, types_, sizes))
    results = []
    for model in (m, other):
        model.model.interaction_blocks[0].train(not training)
        out = model(_data(pos, types_, sizes)).out["SchNet"]
        if training:
            assert not _fused(out["forces"])
            ((out["forces"] - target.to(DEV)) ** 2).mean().backward()
        results.append((out["forces"].detach(), _grads(model.model)))
    assert torch.equal(results[0][0], results[1][0]) and results[0][1].keys() == results[1][1].keys()
    _close(results[0][1], results[1][1], 1e-6)
    if training:
        assert "interaction_blocks.0.conv.lin1.weight" not in results[0][1]


@pytest.mark.parametrize("training", [True, False])
def test_a_basis_whose_scale_changes_after_a_call(training):
    sizes = [23, 40]
    net, pos, types_, batch, target = _setup("expnormal", 32, 9.0, 2, sizes, 128, 22)
    m = bnn.GradientsOut(net.to(DEV), "forces").train(training)
    before = m(_data(pos, types_, sizes)).out["SchNet"]["forces"].detach()
    net.rbf_layer.alpha *= 0.8
    got = m(_data(pos, types_, sizes)).out["SchNet"]["forces"].detach()
    fresh = copy.deepcopy(m)(_data(pos, types_, sizes)).out["SchNet"]["forces"].detach()
    assert torch.equal(got, fresh) and not torch.allclose(got, before, rtol=1e-2)
