"""Mixture-of-experts building blocks with expert parallelism (Mixtral-style top-k routing).

The reference has no MoE support (only an ``"expert"`` axis name in a mesh test, tests/test_mpmd_mesh.py:71).
Routing here is capacity based so that every shape in the captured step is static:

    probs   = softmax(x W_r^T)                       [T, E]
    top-k   → expert ids, weights renormalised over the k picks; aux = E * Σ_e f_e · P_e (load balancing)
    dispatch: token t's copy for expert e goes to slot (number of earlier tokens routed to e); copies beyond
              the capacity C are dropped                → buffer [E, C, d]
    all-to-all over the expert axis: rank r keeps experts [r·E_l, (r+1)·E_l)           → [E_l, ep·C, d]
    expert FFN (SwiGLU) per local expert — equal-sized groups, one tcgen05 GEMM per expert and projection
    all-to-all back, combine: y_t = Σ_k w_{t,k} · out[e_{t,k}, slot_{t,k}]

With expert parallelism the two exchanges are the ops ``b200moe::dispatch_a2a`` (permutation into slots +
all-to-all) and ``b200moe::combine_a2a`` (all-to-all back + weighted gather-sum); each is the other's
transpose, which is how their backward is written.  On GPUs with fused collectives enabled they run as one
peer-memory kernel each (``jaxpp_b200.parallel.fused_moe``), otherwise as index ops around
``b200moe::all_to_all`` (NCCL / gloo).
"""
from __future__ import annotations

import torch
import torch.distributed as dist
from torch import Tensor

from ..ops import core as ops
from . import tp as tpmod

_lib = torch.library.Library("b200moe", "DEF")


def _all_to_all_impl(x: Tensor, axis: str) -> Tensor:
    """x: [n, ...] — block q goes to rank q of the axis; returns [n, ...] with block q received from rank q."""
    n = tpmod.axis_size(axis)
    if n == 1:
        return x
    x = x.contiguous()
    out = torch.empty_like(x)
    dist.all_to_all_single(out, x, group=tpmod._group(axis))
    return out


_lib.define("all_to_all(Tensor x, str axis) -> Tensor")
_lib.impl("all_to_all", _all_to_all_impl, "CompositeExplicitAutograd")
torch.library.register_fake("b200moe::all_to_all", lambda x, axis: torch.empty_like(x))
torch.library.register_autograd(
    "b200moe::all_to_all",
    lambda ctx, g: (torch.ops.b200moe.all_to_all(g.contiguous(), ctx.axis), None),
    setup_context=lambda ctx, inputs, output: setattr(ctx, "axis", inputs[1]),
)


# ---- dispatch / combine fused with the expert-parallel exchange ------------------------------------------------------
def _use_fused(x: Tensor) -> bool:
    from ..utils import config

    if not (x.is_cuda and config.use_fused_collectives.value and config.use_native_kernels.value):
        return False
    from . import fused_moe

    return fused_moe.supported(x)


def _dispatch_a2a_impl(x, dest, scale, n_experts: int, capacity: int, top_k: int, axis: str):
    """x [T, d]; dest [T*k] slot (expert * C + position, E*C = dropped); scale [T*k] or None.
    Returns [E_l, ep*C, d]: for every local expert, the slots of rank 0's tokens, then rank 1's, ..."""
    ep = tpmod.axis_size(axis)
    d = x.shape[-1]
    e_local = n_experts // ep
    if ep > 1 and _use_fused(x):
        from . import fused_moe

        n_slots = n_experts * capacity
        picks = torch.arange(dest.numel(), device=x.device, dtype=torch.int32)
        inv = torch.full((n_slots + 1,), -1, dtype=torch.int32, device=x.device)
        inv[dest] = picks // top_k
        slot_scale = None
        if scale is not None:
            slot_scale = torch.zeros(n_slots + 1, dtype=torch.float32, device=x.device)
            slot_scale[dest] = scale.float()
        return fused_moe.dispatch(x, inv, slot_scale, n_experts, capacity, axis)
    src = x.repeat_interleave(top_k, dim=0)
    if scale is not None:
        src = (src.float() * scale.float().unsqueeze(-1)).to(x.dtype)
    buf = torch.zeros(n_experts * capacity + 1, d, dtype=x.dtype, device=x.device)
    buf = buf.index_add(0, dest, src)[:-1]
    if ep == 1:
        return buf.view(n_experts, capacity, d)
    buf = _all_to_all_impl(buf.view(ep, e_local * capacity, d), axis)   # block q from rank q
    return buf.view(ep, e_local, capacity, d).transpose(0, 1).reshape(e_local, ep * capacity, d)


def _combine_a2a_impl(y, dest, weights, n_experts: int, capacity: int, top_k: int, axis: str, want_picked: bool):
    """y [E_l, ep*C, d] -> (out [T, d], picked [T*k, d] or an empty tensor)."""
    ep = tpmod.axis_size(axis)
    d = y.shape[-1]
    e_local = n_experts // ep
    T = dest.numel() // top_k
    if ep > 1 and _use_fused(y):
        from . import fused_moe

        out, picked = fused_moe.combine(y, dest.to(torch.int32), None if weights is None else weights.float().contiguous(),
                                        n_experts, capacity, top_k, axis, want_picked)
        return out, picked if picked is not None else y.new_empty(0)
    if ep > 1:
        y = y.view(e_local, ep, capacity, d).transpose(0, 1).reshape(ep, e_local * capacity, d)
        y = _all_to_all_impl(y.contiguous(), axis)
    flat = torch.cat([y.reshape(n_experts * capacity, d), torch.zeros(1, d, dtype=y.dtype, device=y.device)], 0)
    picked = flat.index_select(0, dest)
    w = weights.float() if weights is not None else torch.ones(dest.numel(), dtype=torch.float32, device=y.device)
    out = (picked.view(T, top_k, d).float() * w.view(T, top_k, 1)).sum(1).to(y.dtype)
    return out, picked if want_picked else y.new_empty(0)


_lib.define("dispatch_a2a(Tensor x, Tensor dest, Tensor? scale, int n_experts, int capacity, int top_k, str axis) -> Tensor")
_lib.impl("dispatch_a2a", _dispatch_a2a_impl, "CompositeExplicitAutograd")
_lib.define("combine_a2a(Tensor y, Tensor dest, Tensor? weights, int n_experts, int capacity, int top_k, str axis, "
            "bool want_picked) -> (Tensor, Tensor)")
_lib.impl("combine_a2a", _combine_a2a_impl, "CompositeExplicitAutograd")


def _dispatch_fake(x, dest, scale, n_experts, capacity, top_k, axis):
    ep = tpmod.axis_size(axis)
    return x.new_empty(n_experts // ep, ep * capacity, x.shape[-1])


def _combine_fake(y, dest, weights, n_experts, capacity, top_k, axis, want_picked):
    T = dest.numel() // top_k
    return y.new_empty(T, y.shape[-1]), y.new_empty((dest.numel(), y.shape[-1]) if want_picked else (0,))


torch.library.register_fake("b200moe::dispatch_a2a", _dispatch_fake)
torch.library.register_fake("b200moe::combine_a2a", _combine_fake)


def _dispatch_setup(ctx, inputs, output):
    _, dest, scale, ctx.n_experts, ctx.capacity, ctx.top_k, ctx.axis = inputs
    ctx.save_for_backward(dest, scale)


def _dispatch_bwd(ctx, g):
    # the transpose of "scatter rows into slots, scaled" is "gather-sum the slots of each token, scaled";
    # no gradient flows to the scale (it is only used inside the backward of combine)
    dest, scale = ctx.saved_tensors
    dx, _ = torch.ops.b200moe.combine_a2a(g.contiguous(), dest, scale, ctx.n_experts, ctx.capacity, ctx.top_k, ctx.axis, False)
    return dx, None, None, None, None, None, None


def _combine_setup(ctx, inputs, output):
    _, dest, weights, ctx.n_experts, ctx.capacity, ctx.top_k, ctx.axis, ctx.want_picked = inputs
    ctx.has_weights = weights is not None
    ctx.save_for_backward(dest, weights, output[1])


def _combine_bwd(ctx, g_out, g_picked):
    dest, weights, picked = ctx.saved_tensors
    g_out = g_out.contiguous()
    dy = torch.ops.b200moe.dispatch_a2a(g_out, dest, weights, ctx.n_experts, ctx.capacity, ctx.top_k, ctx.axis)
    dw = None
    if ctx.has_weights and ctx.needs_input_grad[2]:
        if not ctx.want_picked:
            raise RuntimeError("combine_a2a needs want_picked=True to differentiate with respect to the weights")
        T = g_out.shape[0]
        dw = (picked.view(T, ctx.top_k, -1).float() * g_out.float().unsqueeze(1)).sum(-1).reshape(-1).to(weights.dtype)
    return dy, None, dw, None, None, None, None, None


torch.library.register_autograd("b200moe::dispatch_a2a", _dispatch_bwd, setup_context=_dispatch_setup)
torch.library.register_autograd("b200moe::combine_a2a", _combine_bwd, setup_context=_combine_setup)


def _route_ref(logits: Tensor, top_k: int):
    """(expert ids [T,k] int64, weights [T,k] fp32, probabilities [T,E] fp32, picks per expert [E] fp32)"""
    probs = torch.softmax(logits.float(), dim=-1)
    top_v, top_i = probs.topk(top_k, dim=-1)
    weights = top_v / top_v.sum(-1, keepdim=True)
    hits = torch.nn.functional.one_hot(top_i, logits.shape[-1]).sum((0, 1)).to(torch.float32)
    return top_i, weights, probs, hits


def _router_impl(logits: Tensor, top_k: int):
    from ..ops import core as _core

    if _native_routing(logits, top_k):
        return _router_native(logits, top_k, False)[:4]
    return _route_ref(logits, top_k)


def _native_routing(logits: Tensor, top_k: int) -> bool:
    return (ops._use_native(logits) and logits.dtype in (torch.float32, torch.bfloat16) and logits.shape[-1] <= 64 and top_k <= 8)


_bound = False


def _native():
    """The native library with the bindings of this module's kernels, and the module that holds it."""
    global _bound
    from ..ops import native

    lib = native.load()
    if not _bound:
        import ctypes

        p, i, f = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
        lib.jpb_router.argtypes = [i, p, p, p, p, p, p, p, f, i, i, i, p]
        lib.jpb_router_scratch_elems.argtypes = [i, i]
        lib.jpb_router_scratch_elems.restype = ctypes.c_longlong
        lib.jpb_router_bwd.argtypes = [i, p, p, p, p, p, p, p, i, i, i, f, p]
        lib.jpb_moe_slots.argtypes = [p, p, p, p, i, i, i, p]
        lib.jpb_moe_dispatch_rows.argtypes = [i, p, p, p, i, i, i, p]
        lib.jpb_moe_combine_rows.argtypes = [i, p, p, p, p, i, i, i, i, p]
        lib.jpb_moe_combine_rows_bwd.argtypes = [i, p, p, p, p, p, p, i, i, i, p]
        _bound = True
    return lib, native


def _aux_scale(T: int, E: int, top_k: int) -> float:
    """aux = E * sum_e (hits_e / (T k)) * mean_t probs[t, e] = _aux_scale * sum_e hits_e * sum_t probs[t, e]"""
    return E / (T * top_k * T) if T else float("nan")


def _router_native(logits: Tensor, top_k: int, want_aux: bool):
    lib, native = _native()
    lg = logits.contiguous()
    T, E = lg.shape
    dev = lg.device
    probs = torch.empty(T, E, dtype=torch.float32, device=dev)
    top_i = torch.empty(T, top_k, dtype=torch.int64, device=dev)
    weights = torch.empty(T, top_k, dtype=torch.float32, device=dev)
    hits = torch.empty(E, dtype=torch.float32, device=dev)
    aux = torch.empty((), dtype=torch.float32, device=dev) if want_aux else None
    part = torch.empty(lib.jpb_router_scratch_elems(T, E), dtype=torch.float32, device=dev) if want_aux else None
    native._check(lib.jpb_router(native._dt(lg), lg.data_ptr(), probs.data_ptr(), top_i.data_ptr(), weights.data_ptr(),
                                 native._p(part), hits.data_ptr(), native._p(aux), _aux_scale(T, E, top_k), T, E, top_k,
                                 native._stream()), "jpb_router", 2 if want_aux else 1)
    return top_i, weights, probs, hits, aux


_lib.define("router(Tensor logits, int top_k) -> (Tensor, Tensor, Tensor, Tensor)")
_lib.impl("router", _router_impl, "CompositeExplicitAutograd")


def _router_fake(logits, top_k):
    T, E = logits.shape
    f32 = dict(dtype=torch.float32, device=logits.device)
    return (torch.empty(T, top_k, dtype=torch.int64, device=logits.device), torch.empty(T, top_k, **f32),
            torch.empty(T, E, **f32), torch.empty(E, **f32))


torch.library.register_fake("b200moe::router", _router_fake)


def _router_setup(ctx, inputs, output):
    ctx.save_for_backward(output[0], output[2])
    ctx.in_dtype = inputs[0].dtype


def _router_bwd(ctx, g_idx, g_w, g_probs, g_hits):
    """weights_j = p_{i_j} / S with S the sum of the picked probabilities; probs = softmax(logits)."""
    top_i, probs = ctx.saved_tensors
    return _logits_grad(top_i, probs, g_w, g_probs).to(ctx.in_dtype), None


def _logits_grad(top_i: Tensor, probs: Tensor, g_w, g_probs) -> Tensor:
    dp = g_probs.float() if g_probs is not None else torch.zeros_like(probs)
    if g_w is not None:
        pv = probs.gather(1, top_i)
        s = pv.sum(-1, keepdim=True)
        gw = g_w.float()
        d_pv = gw / s - (gw * pv).sum(-1, keepdim=True) / (s * s)
        dp = dp.scatter_add(1, top_i, d_pv)
    return probs * (dp - (dp * probs).sum(-1, keepdim=True))


torch.library.register_autograd("b200moe::router", _router_bwd, setup_context=_router_setup)


# The router together with the load-balancing loss: one op each way instead of the router and a dozen small reductions
# and elementwise ops around it (launches, not work, are the cost of routing).
def _route_tokens_impl(logits: Tensor, top_k: int):
    if _native_routing(logits, top_k):
        return _router_native(logits, top_k, True)
    top_i, weights, probs, hits = _route_ref(logits, top_k)
    frac = hits / (top_i.shape[0] * top_k)
    return top_i, weights, probs, hits, logits.shape[-1] * (frac * probs.mean(0)).sum()


def _route_tokens_bwd_impl(top_i: Tensor, probs: Tensor, hits: Tensor, g_w, g_probs, g_aux, like: Tensor) -> Tensor:
    T, E = probs.shape
    k = top_i.shape[1]
    if _native_routing(like, k):
        lib, native = _native()
        gs = [None if g is None else g.float().contiguous() for g in (g_w, g_probs, g_aux)]
        out = torch.empty(T, E, dtype=like.dtype, device=like.device)
        native._check(lib.jpb_router_bwd(native._dt(like), top_i.contiguous().data_ptr(), probs.contiguous().data_ptr(), native._p(gs[0]),
                                         native._p(gs[1]), native._p(gs[2]), hits.contiguous().data_ptr(), out.data_ptr(), T, E, k,
                                         _aux_scale(T, E, k), native._stream()), "jpb_router_bwd")
        return out
    if g_aux is not None:
        d_aux = (g_aux.float() * _aux_scale(T, E, k) * hits).expand_as(probs)
        g_probs = d_aux if g_probs is None else g_probs.float() + d_aux
    return _logits_grad(top_i, probs, g_w, g_probs).to(like.dtype)


_lib.define("route_tokens(Tensor logits, int top_k) -> (Tensor, Tensor, Tensor, Tensor, Tensor)")
_lib.impl("route_tokens", _route_tokens_impl, "CompositeExplicitAutograd")
_lib.define("route_tokens_bwd(Tensor top_i, Tensor probs, Tensor hits, Tensor? g_w, Tensor? g_probs, Tensor? g_aux, Tensor like) -> Tensor")
_lib.impl("route_tokens_bwd", _route_tokens_bwd_impl, "CompositeExplicitAutograd")
torch.library.register_fake("b200moe::route_tokens", lambda logits, top_k: (
    *_router_fake(logits, top_k), torch.empty((), dtype=torch.float32, device=logits.device)))
torch.library.register_fake("b200moe::route_tokens_bwd", lambda top_i, probs, hits, g_w, g_probs, g_aux, like: torch.empty(
    probs.shape, dtype=like.dtype, device=like.device))


def _route_tokens_setup(ctx, inputs, output):
    ctx.save_for_backward(output[0], output[2], output[3], inputs[0])


def _route_tokens_bwd(ctx, g_idx, g_w, g_probs, g_hits, g_aux):
    top_i, probs, hits, logits = ctx.saved_tensors
    return torch.ops.b200moe.route_tokens_bwd(top_i, probs, hits, g_w, g_probs, g_aux, logits), None


torch.library.register_autograd("b200moe::route_tokens", _route_tokens_bwd, setup_context=_route_tokens_setup)


def route(x: Tensor, w_router: Tensor, top_k: int):
    """Returns (expert ids [T,k] int64, weights [T,k] fp32, aux loss scalar fp32).  Softmax, top-k, renormalised
    weights and the load-balancing loss come from one op (``b200moe::route_tokens``)."""
    top_i, weights, _, _, aux = torch.ops.b200moe.route_tokens(ops.linear(x, w_router, None), top_k)
    return top_i, weights, aux


def slots_for(top_i: Tensor, n_experts: int, capacity: int):
    """Flat destination index (expert * C + position) of every (token, pick); dropped picks map to the dump
    row ``E * C``.  Position = how many earlier (token-major) picks chose the same expert."""
    dest, keep, _ = slots_and_counts(top_i, n_experts, capacity)
    return dest, keep


def slots_and_counts(top_i: Tensor, n_experts: int, capacity: int):
    """:func:`slots_for` plus ``counts`` [E] int32: how many slots of each expert this device's tokens fill."""
    flat = top_i.reshape(-1)
    # running count of picks per expert, scanned along the CONTIGUOUS dimension of an [E, picks] int32 matrix: the same
    # scan down the rows of a [picks, E] int64 one-hot matrix took 3.2 ms per call on the GPU (15 % of a Mixtral step)
    onehot_t = (flat[None, :] == torch.arange(n_experts, device=flat.device, dtype=flat.dtype)[:, None]).to(torch.int32)
    running = onehot_t.cumsum(1, dtype=torch.int32)                   # [E, picks]
    pos = (running.gather(0, flat[None, :]).squeeze(0) - 1).to(flat.dtype)
    keep = pos < capacity
    dest = torch.where(keep, flat * capacity + pos, torch.full_like(flat, n_experts * capacity))
    counts = running[:, -1].clamp(max=capacity).to(torch.int32)
    return dest, keep, counts


def dispatch(x: Tensor, dest: Tensor, n_experts: int, capacity: int, top_k: int) -> Tensor:
    """[T, d] → [E, C, d]; every kept (token, pick) copies the token's row into its slot."""
    d = x.shape[-1]
    src = x.repeat_interleave(top_k, dim=0)
    buf = torch.zeros(n_experts * capacity + 1, d, dtype=x.dtype, device=x.device)
    buf = buf.index_add(0, dest, src)
    return buf[:-1].view(n_experts, capacity, d)


def combine(y_buf: Tensor, dest: Tensor, weights: Tensor, top_k: int) -> Tensor:
    """[E, C, d] → [T, d]: weighted sum of each token's picks (dropped picks contribute zero)."""
    E, C, d = y_buf.shape
    flat = torch.cat([y_buf.reshape(E * C, d), torch.zeros(1, d, dtype=y_buf.dtype, device=y_buf.device)], 0)
    picked = flat.index_select(0, dest).view(-1, top_k, d)
    return (picked.float() * weights.unsqueeze(-1)).sum(1).to(y_buf.dtype)


# ---- the same three steps as kernels, where the experts are on this device -------------------------------------------
# ``inv`` [E * C] int32 names the pick that fills each slot (-1: none), so that both directions are gathers: a slot's row
# is written once, zeros included, and no gradient is accumulated with atomics.
def _slots_impl(top_i: Tensor, n_experts: int, capacity: int):
    n = top_i.numel()
    if ops._use_native(top_i) and top_i.dtype == torch.int64 and n_experts <= 64 and n_experts * capacity < 2 ** 31:
        lib, native = _native()
        flat = top_i.contiguous()
        dest = torch.empty(n, dtype=torch.int64, device=flat.device)
        inv = torch.empty(n_experts * capacity, dtype=torch.int32, device=flat.device)
        counts = torch.empty(n_experts, dtype=torch.int32, device=flat.device)
        native._check(lib.jpb_moe_slots(flat.data_ptr(), dest.data_ptr(), inv.data_ptr(), counts.data_ptr(), n, n_experts, capacity,
                                        native._stream()), "jpb_moe_slots")
        return dest, inv, counts
    dest, _, counts = slots_and_counts(top_i, n_experts, capacity)
    inv = torch.full((n_experts * capacity + 1,), -1, dtype=torch.int32, device=dest.device)
    inv[dest] = torch.arange(n, device=dest.device, dtype=torch.int32)
    return dest, inv[:-1].clone(), counts


def _rows_native(t: Tensor, *others) -> bool:
    return (ops._use_native(t) and t.dtype in (torch.float32, torch.bfloat16) and t.shape[-1] % (16 // t.element_size()) == 0
            and all(o is None or o.dtype == torch.float32 for o in others))


def _row_operand(t: Tensor) -> Tensor:
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _dispatch_rows_impl(x: Tensor, dest: Tensor, inv: Tensor, top_k: int) -> Tensor:
    slots, d = inv.numel(), x.shape[-1]
    if _rows_native(x):
        lib, native = _native()
        x = _row_operand(x)
        out = torch.empty(slots, d, dtype=x.dtype, device=x.device)
        native._check(lib.jpb_moe_dispatch_rows(native._dt(x), x.data_ptr(), inv.contiguous().data_ptr(), out.data_ptr(), slots, d, top_k,
                                           native._stream()), "jpb_moe_dispatch_rows")
        return out
    rows = x.index_select(0, (inv.clamp(min=0) // top_k).long())
    return torch.where((inv >= 0).unsqueeze(-1), rows, torch.zeros_like(rows))


def _combine_rows_impl(y: Tensor, dest: Tensor, inv: Tensor, weights, top_k: int) -> Tensor:
    slots, d = y.shape
    T = dest.numel() // top_k
    if _rows_native(y, weights):
        lib, native = _native()
        y = _row_operand(y)
        w = None if weights is None else weights.contiguous()
        out = torch.empty(T, d, dtype=y.dtype, device=y.device)
        native._check(lib.jpb_moe_combine_rows(native._dt(y), y.data_ptr(), dest.contiguous().data_ptr(), native._p(w), out.data_ptr(), T, d,
                                          top_k, slots, native._stream()), "jpb_moe_combine_rows")
        return out
    flat = torch.cat([y, torch.zeros(1, d, dtype=y.dtype, device=y.device)], 0)
    picked = flat.index_select(0, dest).view(T, top_k, d).float()
    return (picked if weights is None else picked * weights.view(T, top_k, 1)).sum(1).to(y.dtype)


def _combine_rows_bwd_impl(g: Tensor, y: Tensor, dest: Tensor, inv: Tensor, weights: Tensor, top_k: int):
    slots, d = y.shape
    T = dest.numel() // top_k
    if _rows_native(y, weights) and g.dtype == y.dtype:
        lib, native = _native()
        g, y, w = _row_operand(g), _row_operand(y), weights.contiguous()
        dy = torch.empty_like(y)
        dw = torch.zeros(T * top_k, dtype=torch.float32, device=y.device)
        native._check(lib.jpb_moe_combine_rows_bwd(native._dt(y), g.data_ptr(), y.data_ptr(), inv.contiguous().data_ptr(), w.data_ptr(),
                                              dy.data_ptr(), dw.data_ptr(), slots, d, top_k, native._stream()), "jpb_moe_combine_rows_bwd")
        return dy, dw
    flat = torch.cat([y, torch.zeros(1, d, dtype=y.dtype, device=y.device)], 0)
    rows = g.float().repeat_interleave(top_k, 0)
    dw = (flat.index_select(0, dest).float() * rows).sum(-1)
    dy = torch.zeros_like(flat).index_copy(0, dest, (rows * weights.reshape(-1, 1)).to(y.dtype))[:-1].clone()
    return dy, dw.to(weights.dtype)


_lib.define("slots(Tensor top_i, int n_experts, int capacity) -> (Tensor, Tensor, Tensor)")
_lib.impl("slots", _slots_impl, "CompositeExplicitAutograd")
_lib.define("dispatch_rows(Tensor x, Tensor dest, Tensor inv, int top_k) -> Tensor")
_lib.impl("dispatch_rows", _dispatch_rows_impl, "CompositeExplicitAutograd")
_lib.define("combine_rows(Tensor y, Tensor dest, Tensor inv, Tensor? weights, int top_k) -> Tensor")
_lib.impl("combine_rows", _combine_rows_impl, "CompositeExplicitAutograd")
_lib.define("combine_rows_bwd(Tensor g, Tensor y, Tensor dest, Tensor inv, Tensor weights, int top_k) -> (Tensor, Tensor)")
_lib.impl("combine_rows_bwd", _combine_rows_bwd_impl, "CompositeExplicitAutograd")
torch.library.register_fake("b200moe::slots", lambda top_i, n_experts, capacity: (
    torch.empty(top_i.numel(), dtype=torch.int64, device=top_i.device),
    torch.empty(n_experts * capacity, dtype=torch.int32, device=top_i.device),
    torch.empty(n_experts, dtype=torch.int32, device=top_i.device)))
torch.library.register_fake("b200moe::dispatch_rows", lambda x, dest, inv, top_k: x.new_empty(inv.shape[0], x.shape[-1]))
torch.library.register_fake("b200moe::combine_rows", lambda y, dest, inv, weights, top_k: y.new_empty(dest.shape[0] // top_k, y.shape[-1]))
torch.library.register_fake("b200moe::combine_rows_bwd", lambda g, y, dest, inv, weights, top_k: (
    torch.empty_like(y, memory_format=torch.contiguous_format), weights.new_empty(dest.shape[0])))


def _dispatch_rows_setup(ctx, inputs, output):
    _, dest, inv, ctx.top_k = inputs
    ctx.save_for_backward(dest, inv)


def _dispatch_rows_bwd(ctx, g):
    dest, inv = ctx.saved_tensors
    return torch.ops.b200moe.combine_rows(g.contiguous(), dest, inv, None, ctx.top_k), None, None, None


def _combine_rows_setup(ctx, inputs, output):
    y, dest, inv, weights, ctx.top_k = inputs
    ctx.save_for_backward(y if weights is not None else None, dest, inv, weights)


def _combine_rows_bwd(ctx, g):
    y, dest, inv, weights = ctx.saved_tensors
    if weights is None:
        return torch.ops.b200moe.dispatch_rows(g.contiguous(), dest, inv, ctx.top_k), None, None, None, None
    dy, dw = torch.ops.b200moe.combine_rows_bwd(g.contiguous(), y, dest, inv, weights, ctx.top_k)
    return dy, None, None, dw, None


torch.library.register_autograd("b200moe::dispatch_rows", _dispatch_rows_bwd, setup_context=_dispatch_rows_setup)
torch.library.register_autograd("b200moe::combine_rows", _combine_rows_bwd, setup_context=_combine_rows_setup)


def expert_ffn(x: Tensor, w_up: Tensor, w_down: Tensor, counts: Tensor | None = None, seg_rows: int = 0) -> Tensor:
    """x: [E_l, M, d]; w_up: [E_l, 2F, d] ([gate | up]); w_down: [E_l, d, F].  Every local expert has room for the
    same number of slots, so each projection is one grouped tcgen05 GEMM over all local experts.  ``counts``
    [E_l, M / seg_rows] says how many slots at the start of each ``seg_rows``-slot segment are filled (the others hold
    zeros): the GEMMs of the forward and of both gradients skip the tiles made of empty slots."""
    E_l, M, d = x.shape
    h = ops.swiglu(ops.linear_batched(x, w_up, counts, seg_rows).view(E_l * M, -1))
    return ops.linear_batched(h.view(E_l, M, -1), w_down, counts, seg_rows)


def moe_ffn(x: Tensor, p: dict, n_experts: int, top_k: int, capacity_factor: float, ep: int, ep_axis: str):
    """Full MoE feed-forward on this device's tokens ``x`` [T, d].  Returns (y [T, d], aux loss)."""
    T, d = x.shape
    capacity = int(-(-T * top_k * capacity_factor // n_experts))
    capacity = (capacity + 7) // 8 * 8
    from ..utils import config

    top_i, weights, aux = route(x, p["router"], top_k)
    if ep == 1:
        dest, inv, counts = torch.ops.b200moe.slots(top_i, n_experts, capacity)
        counts = counts.view(n_experts, 1) if config.moe_skip_empty_slots.value > 0 else None
        buf = torch.ops.b200moe.dispatch_rows(x, dest, inv, top_k).view(n_experts, capacity, d)
        y = expert_ffn(buf, p["w_up"], p["w_down"], counts, capacity)
        return torch.ops.b200moe.combine_rows(y.reshape(n_experts * capacity, d), dest, inv, weights.reshape(-1), top_k), aux
    dest, _, counts = slots_and_counts(top_i, n_experts, capacity)
    if config.moe_skip_empty_slots.value <= 0:
        counts = None
    buf = torch.ops.b200moe.dispatch_a2a(x, dest, None, n_experts, capacity, top_k, ep_axis)   # [E_l, ep*C, d]
    if counts is not None:
        # every rank tells the owner of each expert how many of its C slots it filled: [ep (source), E_l] -> [E_l, ep]
        counts = torch.ops.b200moe.all_to_all(counts.view(ep, n_experts // ep), ep_axis).t().contiguous()
    y = expert_ffn(buf, p["w_up"], p["w_down"], counts, capacity)
    out, _ = torch.ops.b200moe.combine_a2a(y, dest, weights.reshape(-1), n_experts, capacity, top_k, ep_axis, True)
    return out, aux


def _register_direct_calls():
    """Generated task code calls these implementations without the dispatcher (see ops.core.DIRECT)."""
    from ..ops import core as _core

    _core.DIRECT[torch.ops.b200moe.all_to_all.default] = _all_to_all_impl
    _core.DIRECT[torch.ops.b200moe.dispatch_a2a.default] = _dispatch_a2a_impl
    _core.DIRECT[torch.ops.b200moe.combine_a2a.default] = _combine_a2a_impl
    _core.DIRECT[torch.ops.b200moe.router.default] = _router_impl
    _core.DIRECT[torch.ops.b200moe.route_tokens.default] = _route_tokens_impl
    _core.DIRECT[torch.ops.b200moe.route_tokens_bwd.default] = _route_tokens_bwd_impl
    _core.DIRECT[torch.ops.b200moe.slots.default] = _slots_impl
    _core.DIRECT[torch.ops.b200moe.dispatch_rows.default] = _dispatch_rows_impl
    _core.DIRECT[torch.ops.b200moe.combine_rows.default] = _combine_rows_impl
    _core.DIRECT[torch.ops.b200moe.combine_rows_bwd.default] = _combine_rows_bwd_impl


_register_direct_calls()
