"""The training step of the reference's models (GCN, GIN, GAT) as an explicit sequence of launches.

Forward, loss and backward of one mini-batch of a window in one native call (``csrc/torch_ops.cpp``), with the arithmetic
of the autograd functions in ``layers.py`` and the same draws of torch's generator for the dropout; the gradients land in
the flat buffer.  ``plan`` says whether a model is one of those three as they are -- no subclass, no hooks, every parameter
trained -- and returns the step, or None: then the model runs under autograd."""
from __future__ import annotations

import torch

from fastgl import _ops

from . import layers


def _plain(module) -> bool:
    """No hooks anywhere that an explicit sequence of launches would pass by."""
    if torch.nn.modules.module._global_forward_hooks or torch.nn.modules.module._global_forward_pre_hooks:
        return False
    return _no_hooks(module)


def _no_hooks(m) -> bool:
    if m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks:
        return False
    for child in m._modules.values():
        if child is not None and not _no_hooks(child):
            return False
    return True


def plan(trainer):
    """A function (trainer, fb, b, counts row) -> loss that leaves the gradients in ``trainer.grads``, or None.  (It does not
    hold the trainer: a trainer that is dropped gives its memory back at once.)"""
    model, feat, labels = trainer.model, trainer.feat, trainer.labels
    if (type(model) not in (layers.GCN, layers.GIN, layers.GAT) or not torch.is_tensor(feat) or not feat.is_cuda
            or feat.dtype != torch.float32 or feat.dim() != 2 or feat.stride(1) != 1 or not trainer._plain_labels
            or len(model.layers) != len(trainer.fanouts)):
        return None
    params = list(model.parameters())
    if any(p.dtype != torch.float32 or not p.is_cuda or not p.is_contiguous() for p in params):
        return None
    if type(model) is layers.GAT:
        return _plan_gat(trainer)
    if type(model) is layers.GCN and not trainer.table_direct:
        return None
    conv = layers.GCNConv if type(model) is layers.GCN else layers.GINConv
    if any(type(layer) is not conv for layer in model.layers) or type(model.dropout) is not torch.nn.Dropout:
        return None
    if model.layers[0].weights.size(0) != feat.size(1):
        return None

    def step(trainer, fb, b, counts):
        weights, grads = _step_tensors(trainer, [layer.weights for layer in model.layers])
        p_drop = float(model.dropout.p) if model.training else 0.0
        if weights is None or p_drop >= 1.0 or not _plain(model):
            return None
        L = len(weights)
        if conv is layers.GINConv:
            return _ops.gin_step(feat, fb.nodes, fb.block_indptr, fb.block_src, b, counts, weights, grads, p_drop, labels)
        first = [True] + [bool(layers.gcn_aggregate_first(counts[L - i], counts[L - 1 - i], counts[8 + L - 1 - i], *weights[i].shape))
                          for i in range(1, L)]
        return _ops.gcn_step(feat, fb.nodes, fb.block_indptr, fb.block_src, b, counts, weights, grads, first, p_drop, labels)

    return step


def _plan_gat(trainer):
    model, feat, labels = trainer.model, trainer.feat, trainer.labels
    for layer in model.layers:
        if type(layer) is not layers.GATConv or type(layer.fc) is not torch.nn.Linear or layer.fc.bias is not None:
            return None
        if layer.fc.weight.size(0) > layers._GAT_MAX_DIM:
            return None
    if model.layers[0].fc.weight.size(1) != feat.size(1):
        return None

    def step(trainer, fb, b, counts):
        params = [p for layer in model.layers for p in (layer.fc.weight, layer.attn_l, layer.attn_r)]
        params, grads = _step_tensors(trainer, params)
        if params is None or not _plain(model) or any(layer.training and layer.attn_drop.p > 0 for layer in model.layers):
            return None
        if not all(layer.attention_grad for layer in model.layers):
            trainer.grads.zero()
        return _ops.gat_step(feat, fb.nodes, fb.block_indptr, fb.block_src, b, counts, params, grads,
                             [layer.num_heads for layer in model.layers],
                             [layer.leaky_relu.negative_slope for layer in model.layers],
                             [layer.attention_grad for layer in model.layers], labels)

    return step


def _step_tensors(trainer, params):
    """The parameters without their autograd history and the parts of the flat gradient they fill; (None, None) where a
    parameter is frozen or its gradient is not that part any more."""
    views = trainer.grad_views
    grads = [views.get(id(p)) for p in params]
    if any(g is None or not p.requires_grad or p.grad is None or p.grad.data_ptr() != g.data_ptr() for p, g in zip(params, grads)):
        return None, None
    return [p.detach() for p in params], grads
