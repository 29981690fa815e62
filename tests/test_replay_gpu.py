"""Steps replayed as CUDA graphs against the same steps run op by op: same bits, other buffers on every call."""
import gc
import threading

import pytest
import torch
from torch.utils import _pytree as pytree

import jaxpp_b200 as jp
from jaxpp_b200.models import lm_trainer as lt
from jaxpp_b200.models import transformer as tf
from jaxpp_b200.ops import core as ops
from jaxpp_b200.runtime import replay
from jaxpp_b200.utils import config

pytestmark = pytest.mark.gpu


def _mesh():
    return jp.MpmdMesh.create({"mpmd": 1, "data": 1, "model": 1}, kind="cuda", multi_process=False)


def _tensors(tree):
    leaves = pytree.tree_leaves(tree, is_leaf=lambda x: isinstance(x, jp.MpmdArray))
    return [x.local_tensor() if isinstance(x, jp.MpmdArray) else x for x in leaves]


def _replay(step):
    return next(iter(step._cache.values()))._replay


@pytest.mark.parametrize("inplace,clip", [(True, None), (False, 1.0)])
def test_training_steps(inplace, clip):
    cfg = tf.ModelConfig("llama", vocab=1024, d_model=256, n_layers=2, n_heads=4, n_kv_heads=2, ffn=512, seq=128, n_stages=2)
    schedule, device = jp.Interleaved1F1B(2, 1), torch.device("cuda", 0)
    make = lambda: jp.mpmd_jit_with_loop(lt.make_train_step(cfg, schedule, lt.Hyper(inplace_update=inplace, clip_grad_norm=clip)), _mesh())
    graph, eager = make(), make()
    a, b = lt.init_state(cfg, schedule, device, seed=3), lt.init_state(cfg, schedule, device, seed=3)
    g = torch.Generator().manual_seed(0)
    side = torch.cuda.Stream()
    for i in range(6):
        # distinct tokens: the embedding gradient is then a sum without ties in its order
        tok = torch.stack([torch.randperm(cfg.vocab, generator=g)[:2 * 129].view(2, 129) for _ in range(2)]).to(device)
        batch = tok[:, :, :-1].contiguous(), tok[:, :, 1:].contiguous()
        before = _tensors(a["master"])
        if i == 4:     # a replay on another stream than the last one's
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                a, la = graph(a, *batch)
            torch.cuda.current_stream().wait_stream(side)
        else:
            a, la = graph(a, *batch)
        with config.step_graphs.set(False):
            b, lb = eager(b, *batch)
        for x, y in zip(_tensors((a, la)), _tensors((b, lb))):
            assert torch.equal(x, y)
        same = [x.data_ptr() == y.data_ptr() for x, y in zip(before, _tensors(a["master"]))]
        assert all(same) if inplace else not any(same)
    assert _replay(graph).recording is not None and _replay(eager).recording is None


def _chain(x, w):
    y = x
    for _ in range(6):
        y = torch.tanh(y @ w) + x
    return jp.mark_stage_end((y, y.sum(0), x))


def test_results_do_not_share_buffers_between_calls_and_threads():
    step = jp.mpmd_jit_by_yield(_chain, _mesh())
    w = torch.randn(64, 64, device="cuda") / 8
    xs = [torch.randn(32, 64, device="cuda") for _ in range(24)]
    ref = lambda x, w: [t for t in _chain_eager(x, w)]
    outs = [step(x, w) for x in xs[:8]]
    assert _replay(step).recording is not None
    for x, o in zip(xs, outs):
        got = _tensors(o)
        for t, r in zip(got, ref(x, w)):
            torch.testing.assert_close(t, r, rtol=1e-4, atol=1e-4)
        assert got[2].data_ptr() == x.data_ptr()      # a result that is an input is that input, as op by op
    results: dict = {}

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            results[k] = [_tensors(step(x, w)) for x in xs[8 + 8 * k:16 + 8 * k]]
            torch.cuda.current_stream().synchronize()

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    for k in range(2):
        for x, got in zip(xs[8 + 8 * k:16 + 8 * k], results[k]):
            for t, r in zip(got, ref(x, w)):
                torch.testing.assert_close(t, r, rtol=1e-4, atol=1e-4)


def _chain_eager(x, w):
    y = x
    for _ in range(6):
        y = torch.tanh(y @ w) + x
    return y, y.sum(0), x


def test_calls_that_a_recording_does_not_cover_run_op_by_op():
    step = jp.mpmd_jit_by_yield(_chain, _mesh())
    w = torch.randn(64, 64, device="cuda") / 8
    x = torch.randn(32, 64, device="cuda")
    for _ in range(4):
        step(x, w)
    rec = _replay(step).recording
    assert rec is not None
    replays, run = [0], rec.run
    rec.run = lambda inputs: (replays.__setitem__(0, replays[0] + 1), run(inputs))[1]
    step(x, w)
    assert replays[0] == 1
    strided = torch.randn(64, 32, device="cuda").t()
    with config.moe_skip_empty_slots.set(2):
        got = [_tensors(step(x, w)), _tensors(step(strided, w))]
    got.append(_tensors(step(strided, w)))
    with torch.autocast("cuda", dtype=torch.bfloat16):
        step(x, w)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):      # inside another recording
        inner = _tensors(step(x, w))
    graph.replay()
    torch.cuda.synchronize()
    assert replays[0] == 1
    for t, r in zip(inner, _chain_eager(x, w)):
        torch.testing.assert_close(t, r, rtol=1e-4, atol=1e-4)
    for out, inp in zip(got, (x, strided, strided)):
        for t, r in zip(out, _chain_eager(inp, w)):
            torch.testing.assert_close(t, r, rtol=1e-4, atol=1e-4)
    big = jp.mpmd_jit_by_yield(_chain, _mesh())
    wide = torch.randn(5000, 4096, device="cuda")      # more input than is worth copying
    square = torch.randn(4096, 4096, device="cuda") / 64
    for _ in range(4):
        big(wide, square)
    assert _replay(big).recording is None


def _update_slices(flat, other, m, v, g, step):
    n = flat.shape[0] // 2
    out = []
    for lo, hi in ((8, n), (n, 2 * n)):      # parameters that live in one flat buffer of fp32 state
        _, _, _, lp = ops.adamw(flat[lo:hi], g[lo:hi], m[lo:hi], v[lo:hi], step, 1e-2, 0.9, 0.95, 1e-8, 0.1, 1.0, torch.bfloat16, None, True)
        out.append(lp * 2 + 1)
    return jp.mark_stage_end((*out, flat, other + 1))


@pytest.mark.parametrize("aliased", [False, True])
def test_updates_in_place_of_views_reach_the_callers_buffers(aliased):
    """The step updates slices at an offset of its inputs; with ``aliased`` another input overlaps the updated buffer."""
    step, eager = (jp.mpmd_jit_by_yield(_update_slices, _mesh()) for _ in range(2))
    n = 1024

    def fresh():
        gen = torch.Generator(device="cuda").manual_seed(4)
        buf = torch.randn(4 * n, generator=gen, device="cuda")
        m, g = torch.randn(2, 2 * n, generator=gen, device="cuda").unbind(0)
        v = torch.rand(2 * n, generator=gen, device="cuda")
        other = buf[n:3 * n] if aliased else buf[2 * n:4 * n]
        return buf[:2 * n], other, m.clone(), v, g.clone(), torch.tensor(3, device="cuda")

    a, b = fresh(), fresh()
    for _ in range(6):
        got = _tensors(step(*a))
        with config.step_graphs.set(False):
            want = _tensors(eager(*b))
        for x, y in zip((*got, *a), (*want, *b)):
            assert torch.equal(x, y)
        assert got[2].data_ptr() == a[0].data_ptr()
    assert _replay(step).recording is not None


def test_calls_with_other_shapes_and_types_than_the_recorded_ones():
    step = jp.mpmd_jit_by_yield(_chain, _mesh())
    w = torch.randn(64, 64, device="cuda") / 8
    x = torch.randn(32, 64, device="cuda")
    step(x, w)
    compiled = next(iter(step._cache.values()))
    for _ in range(4):
        compiled(x, w)
    assert compiled._replay.recording is not None
    for dtype, rows in ((torch.float32, 1), (torch.float64, 32), (torch.float32, 48)):
        y, v = torch.randn(rows, 64, dtype=dtype, device="cuda"), w.to(dtype)
        got = _tensors(compiled(y, v))
        for t, r in zip(got, _chain_eager(y, v)):
            assert t.shape == r.shape and t.dtype == r.dtype
            torch.testing.assert_close(t, r, rtol=1e-4, atol=1e-4)


def test_memory_of_all_recordings_is_bounded_with_their_inputs(monkeypatch):
    """One program per shape, 65 MB of inputs each: the limit counts the copies of the inputs and is given back."""
    gc.collect()
    before, limit = replay._pool_bytes[0], replay.MAX_POOL_BYTES + (264 << 20)
    monkeypatch.setattr(replay, "TOTAL_POOL_BYTES", before + limit)
    step = jp.mpmd_jit_by_yield(_chain, _mesh())
    w = torch.randn(4096, 4096, device="cuda") / 64
    for rows in range(8, 80, 8):
        x = torch.randn(rows, 4096, device="cuda")
        for _ in range(4):
            got = _tensors(step(x, w))
        for t, r in zip(got, _chain_eager(x, w)):
            torch.testing.assert_close(t, r, rtol=1e-3, atol=1e-3)
    recs = [c._replay.recording for c in step._cache.values() if c._replay.recording is not None]
    copies, kept = sum(s.nbytes for rec in recs for s in rec.static), replay._pool_bytes[0] - before
    assert recs and copies < kept <= limit and len(recs) < 9
    del recs, step, got
    gc.collect()
    assert replay._pool_bytes[0] == before


def test_the_flag_holds_for_each_call():
    w, x = torch.randn(64, 64, device="cuda") / 8, torch.randn(32, 64, device="cuda")
    step = jp.mpmd_jit_by_yield(_chain, _mesh())
    for on, recorded in ((True, False), (True, False), (False, False), (False, False), (True, True)):
        with config.step_graphs.set(on):
            step(x, w)
        assert (_replay(step).recording is not None) == recorded
    replays, run = [0], _replay(step).recording.run
    _replay(step).recording.run = lambda inputs: (replays.__setitem__(0, replays[0] + 1), run(inputs))[1]
    with config.step_graphs.set(False):
        step(x, w)
    assert replays[0] == 0
    late = jp.mpmd_jit_by_yield(_chain, _mesh())
    with config.step_graphs.set(False):      # a warm-up without graphs
        late(x, w)
    for _ in range(3):
        late(x, w)
    assert _replay(late).recording is not None
