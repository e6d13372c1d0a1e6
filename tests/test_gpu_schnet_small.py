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
