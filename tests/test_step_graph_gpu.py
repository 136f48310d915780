"""Captured training / validation passes against the ordinary ones: the same bits, whatever happens in between (GPU)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(graphs: bool, monkeypatch=None, **kw):
    from scaffold_b200.models.unet import UNet
    from scaffold_b200.ops.optim import FusedClipAdam
    from scaffold_b200.train.engine import TrainEngine
    torch.manual_seed(3)
    model = UNet(3, 5, layers=2, base_width=32).cuda()
    eng = TrainEngine(model, FusedClipAdam(model.parameters(), lr=1e-3), 5, torch.device("cuda"), **kw)
    if not graphs:
        eng._graphs.get = lambda *a, **k: None
    return eng


def _batch(seed, n=2, edge=(16, 24, 16), device="cuda"):
    g = torch.Generator().manual_seed(seed)
    x = torch.rand((n, 3, *edge), generator=g)
    y = torch.randint(0, 5, (n, *edge), generator=g, dtype=torch.int16)
    return (x.cuda(), y.cuda()) if device == "cuda" else (x.pin_memory(), y.pin_memory())


def _captured(eng):
    from scaffold_b200.train.step_graph import _Pass
    return [k for k, v in eng._graphs._passes.items() if isinstance(v, _Pass)]


def test_replayed_steps_are_the_ordinary_steps_bit_for_bit():
    a, b = _engine(True), _engine(False)
    side = torch.cuda.Stream()
    kept = []
    for i in range(14):
        batch = _batch(i, device="cpu" if i in (5, 6) else "cuda")
        if i == 7:      # another learning rate
            for e in (a, b):
                e.optimizer.param_groups[0]["lr"] = 3e-4
        if i == 8:      # weights changed behind the optimizer's back
            for e in (a, b):
                e.model.load_state_dict({k: v * 0.9 for k, v in e.model.state_dict().items()})
        if i == 9:      # gradients dropped by the caller
            for e in (a, b):
                e.model.zero_grad(set_to_none=True)
        if i == 10:     # a ragged last batch, then validation between training steps
            small = _batch(100, n=1)
            assert torch.equal(a.step(*small), b.step(*small))
            for _ in range(4):
                for s, t in zip(a.eval_step(*batch), b.eval_step(*batch)):
                    assert torch.equal(s, t)
        if i == 11:
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                la = a.step(*batch)
            torch.cuda.current_stream().wait_stream(side)
        else:
            la = a.step(*batch)
        lb = b.step(*batch)
        kept.append((la, lb))
        assert torch.equal(a.last_ce, b.last_ce) and torch.equal(a.last_dice, b.last_dice)
        assert torch.equal(a.flat.grad, b.flat.grad) and torch.equal(a.flat.data, b.flat.data), i
    assert len(_captured(a)) == 2 and not _captured(b)
    for la, lb in kept:  # a returned loss stays the caller's after later steps
        assert torch.equal(la, lb)


def test_a_changed_model_leaves_the_captured_pass():
    eng = _engine(True)
    batch = _batch(1)
    for _ in range(4):
        eng.step(*batch)
    assert _captured(eng)
    calls = []
    h = eng.model.down_list[0].register_forward_hook(lambda *a: calls.append(1))
    eng.step(*batch)
    assert len(calls) == 1 and not _captured(eng)   # the hook ran: the ordinary pass did
    eng.step(*batch)
    eng.step(*batch)
    assert len(calls) == 3 and not _captured(eng)
    h.remove()
    for _ in range(3):
        eng.step(*batch)
    assert len(calls) == 3 and _captured(eng)
    eng.model.up_list[0].conv.double_conv[1].eps = 1e-3
    eng.step(*batch)
    assert not _captured(eng)


def test_class_weights_are_read_at_replay_and_evaluation_follows_new_weights():
    cw = torch.tensor([1.0, 5.0, 5.0, 5.0, 5.0], device="cuda")
    a, b = _engine(True, class_weights=cw), _engine(False, class_weights=cw)
    batch = _batch(2)
    for i in range(6):
        if i == 4:
            cw.mul_(2.0)
            for e in (a, b):
                with torch.no_grad():
                    for p in e.model.parameters():
                        p.add_(0.01)
        for s, t in zip(a.eval_step(*batch), b.eval_step(*batch)):
            assert torch.equal(s, t), i
    assert _captured(a)


@pytest.mark.parametrize("what", ["saved_tensors", "function_mode", "dual_level"])
def test_an_observer_of_operations_sees_the_ordinary_pass(what):
    from contextlib import nullcontext

    from torch.overrides import TorchFunctionMode
    class Mode(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    eng = _engine(True)
    batch = _batch(0)
    for _ in range(4):
        eng.step(*batch)
    assert _captured(eng)
    packed = []
    ctx = {"saved_tensors": lambda: torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(1), t)[1], lambda t: t),
           "function_mode": Mode, "dual_level": torch.autograd.forward_ad.dual_level}[what]
    for manager, usable in ((ctx, False), (nullcontext, True)):
        with manager():
            assert (eng._graphs.get(eng, *batch, train=True) is not None) is usable
    with ctx():
        eng.step(*batch)
    assert bool(packed) is (what == "saved_tensors")


@pytest.mark.parametrize("how", ["deepcopy", "assign"])
def test_validation_of_a_copied_model_follows_its_weights(how):
    """The operand copies of a model that was copied, or got new parameters, after a first pass."""
    import copy

    from scaffold_b200.models.unet import UNet
    from scaffold_b200.ops.optim import FusedClipAdam
    from scaffold_b200.train.engine import TrainEngine
    dev = torch.device("cuda")

    def make(graphs):
        torch.manual_seed(3)
        model = UNet(3, 5, layers=2, base_width=32).cuda()
        TrainEngine(model, FusedClipAdam(model.parameters(), lr=1e-3), 5, dev).eval_step(*_batch(0))
        if how == "deepcopy":
            model = copy.deepcopy(model)
        else:
            model.load_state_dict({k: v.clone() for k, v in model.state_dict().items()}, assign=True)
        eng = TrainEngine(model, FusedClipAdam(model.parameters(), lr=1e-3), 5, dev)
        if not graphs:
            eng._graphs.get = lambda *a, **k: None
        return eng

    a, b = make(True), make(False)
    batch = _batch(1)
    for i in range(12):
        if i in (5, 8):
            for e in (a, b):
                e.step(*batch)
        if i == 10:
            for e in (a, b):
                e.model.load_state_dict({k: v * 0.9 for k, v in e.model.state_dict().items()})
        for s, t in zip(a.eval_step(*batch), b.eval_step(*batch)):
            assert torch.equal(s, t), i
    assert _captured(a) and not _captured(b)


def test_copies_that_nothing_would_renew_keep_the_ordinary_pass():
    from scaffold_b200.ops import conv3d as c3
    a, b = _engine(True), _engine(False)
    batch = _batch(1)
    for e in (a, b):
        e.eval_step(*batch)
    conv = a.model.up_list[0].conv.double_conv[3]
    c3._PACK_REGISTRY.discard(conv._cache)
    conv._cache.conv3 = lambda w, *r: (type(conv._cache).conv3(conv._cache, w, *r),
                                       c3._PACK_REGISTRY.discard(conv._cache))[0]
    for i in range(8):
        if i == 6:
            for e in (a, b):
                e.step(*batch)
        for s, t in zip(a.eval_step(*batch), b.eval_step(*batch)):
            assert torch.equal(s, t), i
    assert not _captured(a)


def test_a_failed_capture_leaves_no_copies_marked_fresh(monkeypatch):
    """Packing that was recorded but never run must not count as done."""
    a, b = _engine(True), _engine(False)
    batch = _batch(1)
    for e in (a, b):
        for _ in range(2):
            e.step(*batch)
    ordinary = type(a).forward_loss

    def failing(self, *args):
        for m in self.model.modules():
            if getattr(m, "_cache", None) is not None:
                m._cache._fresh, m._cache._bufs = set(), {}   # the pass packs for itself
        ordinary(self, *args)
        raise RuntimeError("out of memory, say")

    from scaffold_b200.train import step_graph as sg
    with monkeypatch.context() as m:
        m.setattr(type(a), "forward_loss", failing)
        m.setattr(sg, "_OWN_FUNCTIONS", sg._functions(type(a)))
        stream = torch.cuda.current_stream()
        assert a._graphs.get(a, *batch, train=True) is None
        assert torch.cuda.current_stream() == stream
    for _ in range(3):
        assert torch.equal(a.step(*batch), b.step(*batch))
        assert torch.equal(a.flat.data, b.flat.data)


def test_another_model_in_the_engine_leaves_the_captured_passes():
    import copy
    a, b = _engine(True), _engine(False)
    batch = _batch(4)
    for _ in range(4):
        for e in (a, b):
            e.step(*batch)
            e.eval_step(*batch)
    assert len(_captured(a)) == 2
    averaged = copy.deepcopy(a.model)
    with torch.no_grad():
        for p in averaged.parameters():
            p.mul_(0.7)
    models = a.model, b.model
    a.model = b.model = averaged
    for _ in range(5):
        for s, t in zip(a.eval_step(*batch), b.eval_step(*batch)):
            assert torch.equal(s, t)
    a.model, b.model = models
    for _ in range(4):
        assert torch.equal(a.step(*batch), b.step(*batch))
        for s, t in zip(a.eval_step(*batch), b.eval_step(*batch)):
            assert torch.equal(s, t)
    assert len(_captured(a)) == 2


def _counting(fn, seen):
    def call(*args, **kwargs):
        seen.append(1)
        return fn(*args, **kwargs)
    return call


@pytest.mark.parametrize("what", ["block", "head", "padded", "features", "forward_loss", "eval_pass", "to_device"])
@pytest.mark.parametrize("when", ["before", "after"])
def test_a_replaced_function_runs_on_every_pass(what, when):
    eng = _engine(True)
    batch = _batch(1)
    owner, name = {"block": (eng.model.down_list[1], "forward"), "head": (eng.model.up_list[-1].conv, "forward_padded"),
                   "padded": (eng.model, "forward_padded_logits"), "features": (eng.model, "features"),
                   "forward_loss": (eng, "forward_loss"), "eval_pass": (eng, "_eval_pass"),
                   "to_device": (eng, "to_device")}[what]

    def passes(n):
        for _ in range(n):
            eng.eval_step(*batch)
    if when == "after":
        passes(4)
        assert len(_captured(eng)) == 1
    seen = []
    setattr(owner, name, _counting(getattr(owner, name), seen))   # a plain function on the instance
    passes(5)
    assert len(seen) == 5
    delattr(owner, name)
    passes(4)
    assert len(seen) == 5 and len(_captured(eng)) == 1


@pytest.mark.parametrize("setting", ["compiled", "dilation", "attribute", "class_function", "submodule", "subclass"])
def test_what_a_pass_depends_on_ends_the_replays(setting, monkeypatch):
    from scaffold_b200.ops import conv3d as c3
    eng = _engine(True)
    batch = _batch(1)
    for _ in range(4):
        eng.eval_step(*batch)
    assert _captured(eng)
    conv = eng.model.down_list[1].maxpool_conv[1].double_conv
    if setting == "compiled":
        conv[0]._compiled_call_impl = conv[0]._call_impl   # what Module.compile() sets
    elif setting == "dilation":
        conv[0].dilation = (2, 2, 2)
    elif setting == "attribute":
        conv[1].num_groups = 4
    elif setting == "class_function":
        monkeypatch.setattr(c3.Conv3d, "_cuda_forward", _counting(c3.Conv3d._cuda_forward, []))
    elif setting == "submodule":
        conv[2] = torch.nn.Dropout3d(0.5)
    else:
        class Mine(type(eng)):
            def forward_loss(self, *args):
                return super().forward_loss(*args)
        eng.__class__ = Mine
    assert eng._graphs.get(eng, *batch, train=False) is None
    if setting in ("submodule", "subclass", "compiled"):   # ... and there are none of such a model
        with torch.no_grad():
            assert all(eng._graphs.get(eng, *batch, train=False) is None for _ in range(5))


@pytest.mark.parametrize("captured_first", [False, True])
def test_a_batch_that_needs_a_gradient_gets_it(captured_first):
    a, b = _engine(True), _engine(False)
    for _ in range(4 if captured_first else 0):
        for e in (a, b):
            e.step(*_batch(0))
    for i in range(5):
        grads = []
        for e in (a, b):
            x, y = _batch(i)
            x.requires_grad_()
            e.step(x, y)
            grads.append(x.grad)
        assert grads[0] is not None and torch.equal(*grads)
    for _ in range(5):   # the ordinary batches around it are replayed, from buffers that are no part of a graph
        assert torch.equal(a.step(*_batch(9)), b.step(*_batch(9)))
    assert len(_captured(a)) == 1
    static = a._graphs._passes[_captured(a)[0]].images
    assert static.is_leaf and not static.requires_grad
    assert torch.equal(a.flat.data, b.flat.data)
    x, y = _batch(3)
    for i in range(8):
        x.requires_grad_(i % 2 == 0)
        assert torch.equal(a.eval_step(x, y)[0], b.eval_step(x, y)[0])
    assert len(_captured(a)) == 2


def test_validation_inside_and_outside_of_inference_mode():
    a, b = _engine(True), _engine(False)
    batch = _batch(2)
    for i in range(14):
        with torch.inference_mode(i < 4 or i % 3 == 0):
            got, want = a.eval_step(*batch), b.eval_step(*batch)
            assert [t.is_inference() for t in got] == [t.is_inference() for t in want]
            for s, t in zip(got, want):
                assert torch.equal(s, t), i
        if i == 8:
            for e in (a, b):
                e.step(*batch)
    assert len(_captured(a)) == 1


def test_replayed_passes_count_in_the_region_totals():
    from scaffold_b200.utils import perf
    totals = []
    for graphs in (True, False):
        eng = _engine(graphs)
        before = {k: v["count"] for k, v in perf.region_totals().items()}
        for i in range(6):
            eng.step(*_batch(i))
            eng.eval_step(*_batch(i))
        assert len(_captured(eng)) == 2 * graphs
        totals.append({k: v["count"] - before.get(k, 0) for k, v in perf.region_totals().items()})
    # a capture runs the pass's Python once more
    for name, extra in (("image_to_device", 0), ("predict", 2), ("calculate_loss", 2), ("backward", 0),
                        ("step_and_update", 0)):
        assert totals[0][name] == totals[1][name] + extra, name


def test_captured_passes_keep_a_bounded_share_of_the_memory(monkeypatch):
    from scaffold_b200.train import step_graph as sg
    a, b = _engine(True), _engine(False)
    for i in range(4):
        a.step(*_batch(i)), b.step(*_batch(i))
    (key,) = _captured(a)
    kept = a._graphs._passes[key].bytes
    x, _ = _batch(0)
    maps = x.shape[0] * 32 * x[0, 0].numel() * 2    # the widest map is one of many that backward needs
    assert 8 * maps < kept < 1 << 30
    total = torch.cuda.get_device_properties(0).total_memory
    monkeypatch.setattr(sg, "MEMORY_SHARE", total // (kept + (1 << 20)))   # room for this one, not for two
    for i in range(5):
        assert torch.equal(a.step(*_batch(i, n=4)), b.step(*_batch(i, n=4)))
    assert _captured(a) == [key]
    assert torch.equal(a.step(*_batch(9)), b.step(*_batch(9))) and torch.equal(a.flat.data, b.flat.data)


@pytest.mark.parametrize("where", ["forward", "backward", "validation"])
def test_an_ordinary_pass_that_runs_out_of_memory_gets_that_of_the_captured_ones(where):
    """The allocator's error is made on the host, once, in an ordinary pass of another shape."""
    a, b = _engine(True), _engine(False)
    for i in range(4):
        a.step(*_batch(i)), b.step(*_batch(i))
    assert _captured(a)
    failures = []

    def fail_once(*args):
        if not failures:
            failures.append(1)
            raise torch.OutOfMemoryError("out of memory")

    if where == "backward":
        handle = a.model.down_list[0].double_conv[1].weight.register_hook(fail_once)   # near the end of backward
        assert torch.equal(a.step(*_batch(9, n=1)), b.step(*_batch(9, n=1)))
        handle.remove()
    else:
        handle = a.model.up_list[0].register_forward_hook(fail_once)
        if where == "forward":
            assert torch.equal(a.step(*_batch(9, n=1)), b.step(*_batch(9, n=1)))
        else:
            for s, t in zip(a.eval_step(*_batch(9, n=1)), b.eval_step(*_batch(9, n=1))):
                assert torch.equal(s, t)
        handle.remove()
    assert failures and not _captured(a)
    assert torch.equal(a.flat.grad, b.flat.grad) and torch.equal(a.flat.data, b.flat.data)
    failures.clear()
    handle = a.model.up_list[0].register_forward_hook(fail_once)
    with pytest.raises(torch.OutOfMemoryError):   # nothing left to give back
        a.step(*_batch(9, n=1))
    handle.remove()


def test_a_pass_dropped_while_another_stream_replays_it_keeps_its_buffers():
    a, b = _engine(True), _engine(False)
    batch = _batch(1, edge=(32, 32, 32))
    for e in (a, b):
        for _ in range(4):
            want = e.eval_step(*batch)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    static = a._graphs._passes[_captured(a)[0]].images
    size = static.numel()
    with torch.cuda.stream(side):
        for _ in range(20):
            got = a.eval_step(*batch)
    address = static.data_ptr()
    del static
    a._graphs.__init__()            # dropped with replays pending
    reused = torch.full((size,), 1e9, device="cuda")   # the default stream's next allocation of that size
    assert reused.data_ptr() != address or side.query()
    side.synchronize()
    for s, t in zip(got, want):
        assert torch.equal(s, t)


def test_threads_validate_their_own_batches():
    from concurrent.futures import ThreadPoolExecutor
    a, b = _engine(True), _engine(False)
    batches = [_batch(i) for i in range(4)]
    for _ in range(4):
        a.eval_step(*batches[0])
    assert _captured(a)
    want = [b.eval_step(*x) for x in batches]
    torch.cuda.synchronize()

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            out = [a.eval_step(*batches[i]) for _ in range(40)]
            torch.cuda.current_stream().synchronize()
        return out
    with ThreadPoolExecutor(4) as pool:
        got = list(pool.map(work, range(4)))
    for i in range(4):
        for out in got[i]:
            for s, t in zip(out, want[i]):
                assert torch.equal(s, t)


def test_a_copied_engine_starts_without_captured_passes():
    import copy
    a = _engine(True)
    for i in range(4):
        a.eval_step(*_batch(i))
    assert _captured(a)
    c = copy.deepcopy(a._graphs)
    assert c is not a._graphs and not c._passes and _captured(a)


@pytest.mark.parametrize("train", [True, False])
def test_a_pass_that_reads_a_value_on_the_host_is_never_captured(train, monkeypatch):
    """A capture would end with an error there. A function put in the engine's own place on the class could do so."""
    a, b = _engine(True), _engine(False)
    ordinary = type(a).forward_loss
    seen = []

    def reading(self, *args):
        out = ordinary(self, *args)
        seen.append(float(out[0].detach()))
        return out
    with monkeypatch.context() as m:
        m.setattr(type(a), "forward_loss", reading)
        for i in range(6):
            batch = _batch(i)
            got, want = (e.step(*batch) if train else e.eval_step(*batch)[0] for e in (a, b))
            assert torch.equal(got, want) and not _captured(a) and len(seen) == 2 * (i + 1)
    for i in range(4):
        got, want = (e.step(*_batch(i)) if train else e.eval_step(*_batch(i))[0] for e in (a, b))
        assert torch.equal(got, want)
    assert _captured(a) and torch.equal(a.flat.data, b.flat.data)


def test_an_error_of_the_runtime_inside_a_capture_leaves_the_device_usable(monkeypatch):
    """The stream, the random numbers, the allocator and later captures (the synchronisation is refused, nothing runs)."""
    from scaffold_b200.train import step_graph as sg
    a, b = _engine(True), _engine(False)
    for i in range(2):
        a.step(*_batch(i)), b.step(*_batch(i))
    ordinary = type(a).forward_loss

    def reading(self, *args):
        out = ordinary(self, *args)
        float(out[0].detach())
        return out
    torch.cuda.manual_seed(7)
    want = torch.rand(5, device="cuda"), torch.rand(5, device="cuda")
    torch.cuda.manual_seed(7)
    got = [torch.rand(5, device="cuda")]
    stream = torch.cuda.current_stream()
    with monkeypatch.context() as m:
        m.setattr(type(a), "forward_loss", reading)
        m.setattr(sg, "_OWN_FUNCTIONS", sg._functions(type(a)))
        assert torch.equal(a.step(*_batch(2)), b.step(*_batch(2)))
    assert torch.cuda.current_stream() == stream and not _captured(a)
    got.append(torch.rand(5, device="cuda"))
    assert all(torch.equal(g, w) for g, w in zip(got, want))
    torch.cuda.empty_cache()
    for i in range(5):   # another shape is still captured
        assert torch.equal(a.step(*_batch(i, n=1)), b.step(*_batch(i, n=1)))
    assert len(_captured(a)) == 1 and torch.equal(a.flat.data, b.flat.data)
