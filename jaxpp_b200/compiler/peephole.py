"""Graph rewrites applied to the captured step before it is clustered into tasks.

``fuse_norm_backward_adds``: in a pre-norm residual block the gradient of the block input is the sum of the
normalisation's input gradient and the gradient that arrives over the residual connection.  Autograd emits that as
``norm_bwd`` followed by an ``add`` kernel that re-reads both tensors; the fused op writes the sum in the pass that
produces the first operand.  The sum is rounded exactly as the two separate kernels would round it: this rewrite leaves a
program's results as they are, bit for bit.

``widen_parameter_sums``: with fp32 gradients the sums that are the gradients of biases and norm weights are produced in
the parameters' type and cast by a kernel of their own each.  The ops can leave their fp32 sums as they are.  A program
that gets this rewrite is more exact than the eager step, whose sums are rounded to the parameters' type in between, and no
longer the same bits.
"""
from __future__ import annotations

import operator

import torch
from torch import fx


def _val(n: fx.Node):
    return n.meta.get("val")


def fuse_norm_backward_adds(graph: fx.Graph) -> int:
    from ..ops import core as ops  # noqa: F401  (registers the ops)

    fused = {
        torch.ops.b200.rmsnorm_bwd.default: torch.ops.b200.rmsnorm_bwd_add.default,
        torch.ops.b200.layernorm_bwd.default: torch.ops.b200.layernorm_bwd_add.default,
    }
    order = {n: i for i, n in enumerate(graph.nodes)}
    count = 0
    for n in list(graph.nodes):
        if n.op != "call_function" or n.target not in fused:
            continue
        dx_items = [u for u in n.users if u.op == "call_function" and u.target is operator.getitem and u.args[1] == 0]
        if len(dx_items) != 1 or len(dx_items[0].users) != 1:
            continue
        dx = dx_items[0]
        add = next(iter(dx.users))
        if add.op != "call_function" or add.target is not torch.ops.aten.add.Tensor or add.kwargs or len(add.args) != 2:
            continue
        other = add.args[1] if add.args[0] is dx else add.args[0]
        if not isinstance(other, fx.Node) or other is dx or order[other] > order[n]:
            continue
        a, b = _val(dx), _val(other)
        if a is None or b is None or tuple(a.shape) != tuple(b.shape) or a.dtype != b.dtype:
            continue
        with graph.inserting_before(n):
            new = graph.call_function(fused[n.target], (*n.args, other))
        new.meta = dict(n.meta)
        n.replace_all_uses_with(new)
        add.replace_all_uses_with(dx)
        graph.erase_node(add)
        graph.erase_node(n)
        count += 1
    return count


def _casts_to_fp32(n: fx.Node) -> bool:
    return (n.op == "call_function" and n.target is torch.ops.aten._to_copy.default and len(n.args) == 1
            and dict(n.kwargs) == {"dtype": torch.float32})


def widen_parameter_sums(graph: fx.Graph, keep=()) -> int:
    """``keep``: nodes that are referred to from outside of the graph (results of the step) and stay."""
    from ..ops import core as ops  # noqa: F401  (registers the ops)

    b = torch.ops.b200
    n_args = {b.colsum.default: 1, b.rmsnorm_bwd.default: 4, b.rmsnorm_bwd_add.default: 5, b.layernorm_bwd.default: 5,
              b.layernorm_bwd_add.default: 6}
    count = 0
    for n in list(graph.nodes):
        if n.op != "call_function" or n.target not in n_args or len(n.args) != n_args[n.target] or n.kwargs:
            continue
        if n.target is b.colsum.default:
            sums = [n]
        else:
            items = [u for u in n.users if u.op == "call_function" and u.target is operator.getitem]
            if len(items) != len(n.users):
                continue
            sums = [u for u in items if u.args[1] >= 1]
        if not sums or any(_val(s) is None or _val(s).dtype != torch.bfloat16 or not s.users or not all(_casts_to_fp32(u) and u not in keep for u in s.users)
                           for s in sums) or n in keep or any(s in keep for s in sums):
            continue      # someone wants a sum in its own type
        with graph.inserting_before(n):
            new = graph.call_function(n.target, (*n.args, torch.float32))
        new.meta = dict(n.meta)
        wide = lambda v: v.to(torch.float32)
        if n.target is b.colsum.default:
            new.meta["val"] = wide(_val(n))
            sums = [new]
        elif isinstance(_val(n), (tuple, list)):
            new.meta["val"] = type(_val(n))([v if i == 0 else wide(v) for i, v in enumerate(_val(n))])
        n.replace_all_uses_with(new)
        graph.erase_node(n)
        for s in sums:
            if s is not new:
                s.meta["val"] = wide(_val(s))
            for cast in list(s.users):
                cast.replace_all_uses_with(s)
                graph.erase_node(cast)
        count += 1
    return count
