"""What a module keeps between calls (transfer tables, packed 1x1 weights) follows its parameters."""
import pytest
import torch


def _rel(a, r):
    return float((a.double() - r.double()).norm() / r.double().norm())


def test_inference_tensors_have_no_state():
    from conversenet_b200 import _cabi
    with torch.inference_mode():
        t = torch.zeros(3)
    assert _cabi.host().state(torch.zeros(3), None, t) is None
    assert _cabi.host().state(torch.zeros(3), None) is not None


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_modules_made_in_inference_mode_follow_their_parameters(dtype):
    from conversenet_b200 import Converse2D, ConverseBlock

    def change(m):
        for i, q in enumerate(m.parameters()):
            q.add_(0.05 * (i + 1))

    for make, C in ((lambda: Converse2D(8, 8, 3, padding=1), 8), (lambda: ConverseBlock(64, 64, 3, 1, 1), 64)):
        for fixed in (False, True):
            torch.manual_seed(5)
            ordinary = make().cuda().eval()
            x = torch.randn(2, C, 20, 17, device="cuda").to(dtype)
            with torch.inference_mode():
                m = make().cuda().eval()
                m.load_state_dict(ordinary.state_dict())
                m.fixed_order = ordinary.fixed_order = fixed
                first = m(x)
                change(m)
                second = m(x)
            with torch.no_grad():
                assert torch.equal(first, ordinary(x))
                change(ordinary)
                assert torch.equal(second, ordinary(x))
            assert _rel(second, first) > 1e-3


def _block_step(blk, x):
    with torch.no_grad():
        return blk(x)


def test_copies_and_pickles_start_without_kept_values():
    import copy
    import pickle
    from conversenet_b200 import ConverseBlock
    blk = ConverseBlock(64, 64, 3, 1, 1)
    for kept in (blk._pack, blk._pair_table, blk.conv1[3]._tables):
        kept.last = ("key", "value", None)
        kept.entries["key"] = "value"
    for c in (copy.deepcopy(blk), pickle.loads(pickle.dumps(blk))):
        for kept in (c._pack, c._pair_table, c.conv1[3]._tables):
            assert kept.last is None and not kept.entries
    old = blk.__dict__.copy()          # a module pickled before these attributes existed
    for name in ("_pack", "_pair_table", "fixed_order"):
        del old[name]
    c = ConverseBlock.__new__(ConverseBlock)
    c.__setstate__(old)
    assert c._pack.last is None and c.fixed_order is False


class _FakeHost:
    """Stands in for the native module: streams are numbers, joins are recorded."""

    def __init__(self, capturing=False):
        self.capturing, self.joined = capturing, []

    def ready(self, t, *params):
        self.pinned = params
        return None if self.capturing else "event"

    def join(self, event, *tensors):
        if self.capturing:
            return False
        self.joined.append(event)
        return True


def _state(stream, version=0):
    return version.to_bytes(16, "little") + stream.to_bytes(8, "little")


def test_other_streams_wait_for_a_kept_value_once(monkeypatch):
    from conversenet_b200 import _cabi
    from conversenet_b200._kept import Kept
    host = _FakeHost()
    monkeypatch.setattr(_cabi, "host", lambda: host)
    made = []

    def build():
        made.append(torch.zeros(2))
        return made[-1]

    kept, q = Kept(2), torch.zeros(1)
    for stream in (1, 2, 1, 2, 3):
        assert kept.get(("k", _state(stream)), (q,), build) is made[0]
    assert len(made) == 1 and host.joined == ["event"] * 2
    assert host.pinned == (q,)           # the parameter's storage stays taken while the entry lives
    # bounded; the oldest goes first
    kept.get(("k", _state(1, version=1)), (q,), build)
    kept.get(("k", _state(1, version=2)), (q,), build)
    assert len(kept.entries) == 2 and len(made) == 3
    kept.get(("k", _state(1)), (q,), build)
    assert len(made) == 4


def test_nothing_is_kept_while_capturing(monkeypatch):
    from conversenet_b200 import _cabi
    from conversenet_b200._kept import Kept
    host = _FakeHost(capturing=True)
    monkeypatch.setattr(_cabi, "host", lambda: host)
    kept, q = Kept(2), torch.zeros(1)
    kept.get(("k", _state(1)), (q,), lambda: torch.zeros(2))
    assert kept.last is None and not kept.entries
    host.capturing = False
    value = kept.get(("k", _state(1)), (q,), lambda: torch.zeros(2))
    host.capturing = True
    assert kept.get(("k", _state(2)), (q,), lambda: torch.zeros(2)) is value
    host.capturing = False
    kept.get(("k", _state(2)), (q,), lambda: torch.zeros(2))
    assert host.joined == ["event"]      # the eager call on that stream waits


@pytest.mark.gpu
def test_tables_and_packed_weights_across_streams_and_threads():
    """Tables and packed weights are made behind a long queue of work on one stream; calls on another stream, from
    another thread, may not read them before."""
    import threading
    from conversenet_b200 import Converse2D, ConverseBlock
    torch.manual_seed(11)
    for make, C in ((lambda: Converse2D(128, 128, 5, padding=2), 128), (lambda: ConverseBlock(64, 64, 3, 1, 1), 64)):
        m, twin = make().cuda().eval(), make().cuda().eval()
        twin.load_state_dict(m.state_dict())
        x = torch.randn(2, C, 40, 36, device="cuda")
        busy = torch.randn(4096, 4096, device="cuda")
        with torch.no_grad():
            ref = twin(x)
        for _ in range(3):
            a, b = torch.cuda.Stream(), torch.cuda.Stream()
            with torch.no_grad():
                for q in m.parameters():
                    q.add_(0.0)               # a new version: tables and weights are laid out again
            torch.cuda.synchronize()
            with torch.cuda.stream(a), torch.no_grad():
                for _ in range(20):
                    busy @ busy
                first = m(x)
            got = []

            def other():
                with torch.cuda.stream(b), torch.no_grad():
                    got.append(m(x))

            t = threading.Thread(target=other)
            t.start()
            t.join()
            torch.cuda.synchronize()
            assert torch.equal(first, ref) and torch.equal(got[0], ref)


@pytest.mark.gpu
def test_capture_without_warm_up_and_eager_calls_after_it():
    from conversenet_b200 import ConverseBlock
    torch.manual_seed(12)
    blk, twin = ConverseBlock(64, 64, 3, 1, 1).cuda().eval(), ConverseBlock(64, 64, 3, 1, 1).cuda().eval()
    twin.load_state_dict(blk.state_dict())
    x = torch.randn(1, 64, 24, 20, device="cuda")
    ref = _block_step(twin, x)
    g = torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.graph(g):
        y = blk(x)
    assert torch.equal(_block_step(blk, x), ref)      # before any replay
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, ref)
    assert torch.equal(_block_step(blk, x), ref)


@pytest.mark.gpu
@pytest.mark.parametrize("C", [64, 16])      # the hooked route and the layer-by-layer route
def test_block_keeps_its_gelu_when_another_call_runs_inside(C):
    """Another thread's call of the same block may begin and end while this one is between its layers; a hook that runs
    the block again puts it there."""
    from conversenet_b200 import ConverseBlock
    torch.manual_seed(13)
    blk, twin = ConverseBlock(C, C, 3, 1, 1).cuda().eval(), ConverseBlock(C, C, 3, 1, 1).cuda().eval()
    twin.load_state_dict(blk.state_dict())
    x = torch.randn(1, C, 12, 10, device="cuda")
    depth = [0]

    def again(module, args):
        if depth[0] == 0:
            depth[0] = 1
            _block_step(blk, x)
            depth[0] = 0

    blk.conv1[3].register_forward_pre_hook(again)
    twin.conv1[3].register_forward_pre_hook(lambda module, args: None)
    assert torch.equal(_block_step(blk, x), _block_step(twin, x))


@pytest.mark.gpu
def test_a_call_that_waits_for_the_launch_queue_lets_other_threads_run():
    import threading
    import time
    from conversenet_b200 import Converse2D
    m = Converse2D(8, 8, 3, padding=1).cuda().eval()
    x = torch.randn(1, 8, 16, 16, device="cuda")
    with torch.no_grad():
        m(x)
        torch.cuda.synchronize()
        gaps, stop = [], threading.Event()

        def tick():
            last = time.perf_counter()
            while not stop.is_set():
                time.sleep(0.001)
                now = time.perf_counter()
                gaps.append(now - last)
                last = now

        t = threading.Thread(target=tick)
        t.start()
        torch.cuda._sleep(1_500_000_000)      # about 0.8 s of the GPU's time; the calls behind it fill the launch queue
        t0 = time.perf_counter()
        for _ in range(4000):
            m(x)
        waited = time.perf_counter() - t0
        stop.set()
        t.join()
        torch.cuda.synchronize()
    assert waited > 0.4                       # the queue did fill
    assert sum(g for g in gaps if g > 0.05) < 0.5 * waited


def test_backend_variable_is_read_at_every_call(monkeypatch):
    from conversenet_b200 import Converse2D, _cabi
    m = Converse2D(2, 2, 3)
    for load in (False, True):
        monkeypatch.setattr(_cabi, "_host", _cabi.host() if load else None)
        for value, error in (("pytorch", RuntimeError), ("nope", ValueError), ("", None), ("CUDA", None), (None, None)):
            if value is None:
                monkeypatch.delenv("CONVERSE2D_BACKEND", raising=False)
            else:
                monkeypatch.setenv("CONVERSE2D_BACKEND", value)
            if error is None:
                m._check_backend()
            else:
                with pytest.raises(error):
                    m._check_backend()


@pytest.mark.gpu
def test_a_layer_holds_only_the_tables_its_calls_read():
    from conversenet_b200 import Converse2D, _cabi
    from conversenet_b200 import functional as CF
    lib = _cabi.load()
    torch.manual_seed(14)
    C, k = 16, 5
    for n, scale in ((264, 1), (268, 1), (68, 2), (132, 1)):
        m = Converse2D(C, C, k, scale=scale, padding=2).cuda().eval()
        H = n - 4
        x = torch.randn(4, C, H, H, device="cuda")
        held = lambda: sum(e.value[0].numel() for e in m._tables.entries.values())
        with torch.no_grad():
            four = m(x)
            assert held() == lib.cvb_pair_transfer_bytes(C, n, n)
            one = m(x[1:2])
            assert held() == lib.cvb_pair_transfer_bytes(C, n, n) + lib.cvb_plane_transfer_bytes(C, n, n)
            m(x[:2])
            assert held() == lib.cvb_pair_transfer_bytes(C, n, n) + lib.cvb_plane_transfer_bytes(C, n, n)
            # a table for every batch gives the same results
            table, wf = CF.build_transfer(m.weight, m.bias, scale, m.eps, n, n)
            every = CF.converse2d_forward(x, table, wf, k, scale, 2, "circular")
        assert _rel(every, four) <= 2e-6 and _rel(one, four[1:2]) <= 6e-6      # (268: split TF32 products)
        # a table that a call would read past is refused
        table, wf = CF.build_transfer(m.weight, m.bias, scale, m.eps, n, n, batch=1)
        with pytest.raises(RuntimeError):
            CF.converse2d_forward(x, table, wf, k, scale, 2, "circular", pairs=True)
        if CF.takes_pairs(4, n, n, scale) and n > 136:
            with pytest.raises(RuntimeError):
                CF.converse2d_forward(x, table, wf, k, scale, 2, "circular")


@pytest.mark.gpu
def test_a_captured_graph_holds_the_tables_it_reads():
    from conversenet_b200 import ConverseBlock
    from conversenet_b200.graphs import GraphedForward
    torch.manual_seed(15)
    blk = ConverseBlock(64, 64, 3, 1, 1).cuda().eval()
    x = torch.randn(1, 64, 30, 22, device="cuda")
    ref = _block_step(blk, x)
    g = GraphedForward(blk, x)
    for n in range(12):                  # more sizes than a layer keeps tables for, then new versions of all weights
        _block_step(blk, torch.randn(1, 64, 12 + n, 16, device="cuda"))
    with torch.no_grad():
        for q in blk.parameters():
            q.add_(1.0)
    _block_step(blk, x)
    filler = [torch.full((1 << 20,), float("nan"), device="cuda") for _ in range(16)]
    filler += [torch.full((n,), float("nan"), device="cuda") for n in (1 << 10, 1 << 14, 50000, 1 << 17) for _ in range(32)]
    assert torch.equal(g(x), ref)
    del filler


@pytest.mark.gpu
def test_kernels_at_several_sizes_from_several_threads():
    """The same kernels launched with more and with less shared memory at the same time (the adjoint epilogue's tiles take 52 to
    103 KB here): a small call must not take the permission for more from a large one that is about to launch."""
    import threading
    from conversenet_b200 import Converse2D, _cabi
    from conversenet_b200 import functional as CF
    sizes, failures = (20, 36, 68, 132, 20, 68), []
    start = threading.Barrier(len(sizes))

    def work(n):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                m = Converse2D(2, 2, 7, scale=2, padding=0, padding_mode="circular").cuda()
                table, _ = CF.build_transfer(m.weight, m.bias, 2, 1e-5, n, n)
                g = torch.randn(1, 2, 2 * n, 2 * n, device="cuda")
                torch.cuda.current_stream().synchronize()
                start.wait()
                for _ in range(1000):      # (with a limit of the call's own size four of the six threads failed within 510)
                    _cabi.host().backward(None, g, None, table, m.weight, m.bias, (1, 2, n, n), 2, 0, "circular", 1e-5, True, False)
                torch.cuda.current_stream().synchronize()
        except Exception as e:
            failures.append(e)
    threads = [threading.Thread(target=work, args=(n,)) for n in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[0]
