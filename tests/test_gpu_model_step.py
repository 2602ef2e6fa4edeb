"""GPU test of the training steps without autograd: the same trainer with and without them, over steps of GCN, GIN and GAT
stacks, takes the same losses and parameters."""
import numpy as np
import pytest
import torch

from test_gpu_training import setup_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,feat,hidden,fanouts,dropout", [
    ("gcn", 100, 32, (10, 5), 0.5), ("gcn", 61, 128, (5, 4, 3), 0.0), ("gin", 100, 33, (10, 5), 0.5), ("gin", 30, 16, (6,), 0.0),
    ("gat", 50, 8, (10, 5), 0.5), ("gat-constant", 50, 7, (4, 3), 0.0),
])
def test_steps_without_autograd_equal_the_autograd_steps(kind, feat, hidden, fanouts, dropout):
    from fastgl_b200.layers import GAT, GCN, GIN
    from fastgl_b200.trainer import Trainer
    indptr, indices, x, labels, train = setup_problem(feat_dim=feat, seed=17)
    dev = torch.device("cuda", 0)
    runs = []
    for explicit in (True, False):
        torch.manual_seed(3)
        if kind.startswith("gat"):
            model = GAT(feat, hidden, 7, len(fanouts), dropout=dropout, heads=4, attention_grad=kind == "gat")
        else:
            model = {"gcn": GCN, "gin": GIN}[kind](feat, hidden, 7, len(fanouts), dropout=dropout)
        tr = Trainer(*(torch.from_numpy(t).to(dev) for t in (indptr, indices, x, labels, train)), model.to(dev), list(fanouts),
                     batch_size=200, window=3, lr=1e-3)
        assert tr._model_step is not None
        if not explicit:
            tr._model_step = None
        losses = tr.run_steps(5, read_loss_each_step=True)
        runs.append((losses, [p.detach().clone() for p in model.parameters()], tr.sampled_edges))
    (la, pa, ea), (lb, pb, eb) = runs
    assert ea == eb and np.allclose(la, lb, rtol=1e-5, atol=1e-6)
    for p, q in zip(pa, pb):      # five steps of 1e-3: a gradient near zero may turn a step's sign, most entries agree to rounding
        assert float((p - q).abs().max()) <= 1.1e-2 and float((p - q).norm()) <= 1e-3 * float(q.norm())


def test_a_frozen_parameter_or_a_hook_keeps_the_model_under_autograd():
    from fastgl_b200.layers import GCN
    from fastgl_b200.trainer import Trainer
    indptr, indices, x, labels, train = setup_problem(feat_dim=20, seed=17)
    dev = torch.device("cuda", 0)
    torch.manual_seed(3)
    model = GCN(20, 16, 7, 2, dropout=0.0).to(dev)
    tr = Trainer(*(torch.from_numpy(t).to(dev) for t in (indptr, indices, x, labels, train)), model, [5, 5], batch_size=200, window=2)
    seen = []
    model.layers[1].register_forward_hook(lambda *a: seen.append(1))
    tr.run_steps(2)
    assert len(seen) == 2
