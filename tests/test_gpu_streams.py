"""Normal-mode calls on several streams of one rank: results, and whose memory may be handed out again when.

A delay on one stream lets the host run ahead, so that a tensor dropped too early would be overwritten by what the test allocates
next. Overwritten words are zeros: they would give wrong sums, not addresses outside the tensors."""
import pytest
import torch

from helpers import make_routing, make_tokens

pytestmark = pytest.mark.gpu

T, H, E, K = 300, 1024, 16, 4
DELAY = 100_000_000  # cycles, about 50 ms


def _buffer(nvl=256 << 20):
    from deepep_efa_b200.parallel.virtual import VirtualCluster
    vc = VirtualCluster(1, num_nvl_bytes=nvl, timeout_ms=5000)
    return vc, vc.buffers[0]


def _layout(buf, idx, **how):
    per_rank, _, per_expert, in_rank, ev = buf.get_dispatch_layout(idx, E, **how)
    return dict(num_tokens_per_rank=per_rank, num_tokens_per_expert=per_expert, is_token_in_rank=in_rank, topk_idx=idx), ev


def _delay(stream):
    with torch.cuda.stream(stream):
        torch.cuda._sleep(DELAY)


def _overwrite(shapes, dtype=torch.int32, copies=16):
    return [torch.zeros(s, dtype=dtype, device="cuda") for s in shapes for _ in range(copies)]


@pytest.mark.parametrize("call", ["combine", "cached_dispatch"])
def test_handle_outlives_an_asynchronous_call(call):
    """A handle made on the caller's stream and dropped while the communication stream has yet to read it."""
    vc, buf = _buffer()
    try:
        idx, _ = make_routing(T, E, K, "cuda", seed=1, masked_fraction=0.3)
        x, y = make_tokens(T, H, "cuda", seed=1), None
        lay, _ = _layout(buf, idx)

        def step(handle, **how):
            if call == "combine":
                out, _, ev = buf.combine(y, handle, **how)
            else:
                out, _, _, _, _, ev = buf.dispatch(x, handle=handle, **how)
            return out, ev

        y, _, _, _, handle, _ = buf.dispatch(x, **lay)
        want = step(handle)[0].clone()
        handle = buf.dispatch(x, **lay)[4]
        shapes = [t.shape for t in handle]
        torch.cuda.synchronize()
        _delay(buf.comm_stream)
        out, ev = step(handle, async_finish=True)
        del handle
        keep = _overwrite(shapes)
        ev.current_stream_wait()
        torch.cuda.synchronize()
        buf.check_status()
        assert torch.equal(out, want)
        del keep
    finally:
        vc.destroy()


def test_handle_of_an_asynchronous_call_used_and_dropped_elsewhere():
    """Layout and handle made on the communication stream (or the default one) and read by a direct call on a third stream."""
    vc, buf = _buffer()
    try:
        idx, _ = make_routing(T, E, K, "cuda", seed=2, masked_fraction=0.3)
        x = make_tokens(T, H, "cuda", seed=2)
        lay, _ = _layout(buf, idx)
        y, _, _, _, handle, _ = buf.dispatch(x, **lay)
        want = buf.combine(y, handle)[0].clone()
        for asynchronous in (True, False):
            how = dict(async_finish=True) if asynchronous else {}
            lay, ev = _layout(buf, idx, **how)
            if asynchronous:
                ev.current_stream_wait()
            _, _, _, _, handle, ev = buf.dispatch(x, **lay, **how)
            if asynchronous:
                ev.current_stream_wait()
            shapes = [t.shape for t in handle]
            side = torch.cuda.Stream()
            torch.cuda.synchronize()
            _delay(side)
            with torch.cuda.stream(side):
                out, _, _ = buf.combine(y, handle)
            del handle, lay
            keep = _overwrite(shapes)
            with torch.cuda.stream(buf.comm_stream):
                keep += _overwrite(shapes)
            torch.cuda.synchronize()
            buf.check_status()
            assert torch.equal(out, want), asynchronous
            del keep
    finally:
        vc.destroy()


def test_call_of_another_thread_during_the_wait_for_the_counts():
    """A dispatch waits on the host for its receive counts and lets other threads run; what they launch on another stream comes
    after what the dispatch has launched."""
    import threading
    import time
    vc, buf = _buffer()
    try:
        idx, _ = make_routing(T, E, K, "cuda", seed=3)
        x = make_tokens(T, H, "cuda", seed=3)
        lay, _ = _layout(buf, idx)
        y, _, _, want_counts, handle, _ = buf.dispatch(x, **lay)
        want = buf.combine(y, handle)[0].clone()
        first, second = torch.cuda.Stream(), torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(first):
            torch.cuda._sleep(8 * DELAY)
        started, got = threading.Event(), []

        def waiter():
            with torch.cuda.stream(first):
                started.set()
                got.append(buf.dispatch(x, **lay))

        thread = threading.Thread(target=waiter)
        thread.start()
        started.wait()
        time.sleep(0.05)  # the other thread is waiting for its counts by now
        with torch.cuda.stream(second):
            out, _, _ = buf.combine(y, handle)
        early = second.query()
        thread.join()
        torch.cuda.synchronize()
        buf.check_status()
        assert not early
        assert torch.equal(out, want) and got[0][3] == want_counts and torch.equal(got[0][0], x)
    finally:
        vc.destroy()


def test_calls_of_one_capture_on_two_streams():
    """Inside one capture, a layout on the communication stream and one on the capturing stream share the scratch: they come one
    after the other although nothing else orders them."""
    vc, buf = _buffer()
    try:
        n = 5000  # several CTAs, so that the scratch is used
        idx = [make_routing(n, E, K, "cuda", seed=4 + i, masked_fraction=0.1 * i)[0] for i in range(2)]
        want = [[t.clone() for t in (lay["num_tokens_per_expert"], lay["is_token_in_rank"])] for lay in (_layout(buf, i)[0] for i in idx)]
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            first, ev = _layout(buf, idx[0], async_finish=True)
            second, _ = _layout(buf, idx[1])
            ev.current_stream_wait()
        for _ in range(20):
            graph.replay()
            torch.cuda.synchronize()
            for lay, w in zip((first, second), want):
                assert torch.equal(lay["num_tokens_per_expert"], w[0]) and torch.equal(lay["is_token_in_rank"], w[1])
    finally:
        vc.destroy()


@pytest.mark.parametrize("call", ["dispatch", "combine"])
def test_symmetric_memory_dropped_under_another_stream(call):
    """A direct call still has to write (dispatch) or read (combine) symmetric memory on its stream when the last tensor in it dies
    under another one: what is allocated next must lie elsewhere, or come after the call."""
    vc, buf = _buffer(nvl=64 << 20)
    try:
        idx, _ = make_routing(T, E, K, "cuda", seed=5)
        x = make_tokens(T, H, "cuda", seed=5)
        lay, _ = _layout(buf, idx)
        y, _, _, _, handle, _ = buf.dispatch(x, **lay)
        want = buf.combine(y, handle)[0].clone()
        side = torch.cuda.Stream()
        torch.cuda.synchronize()
        _delay(side)
        with torch.cuda.stream(side):
            if call == "dispatch":
                late = buf.dispatch(x, handle=handle)[0]
            else:
                late = buf.empty_symmetric([T, H], torch.bfloat16)
                late.copy_(y)
                out = buf.combine(late, handle)[0]
        late_at = late.data_ptr()
        del late
        fresh = [buf.empty_symmetric([T, H], torch.bfloat16) for _ in range(4)]
        for f in fresh:
            f.fill_(3.0)
        assert late_at not in [f.data_ptr() for f in fresh]
        torch.cuda.synchronize()
        buf.check_status()
        assert all(bool((f == 3.0).all()) for f in fresh)
        if call == "combine":
            assert torch.equal(out, want)
        # the memory comes back once the call is over
        del fresh
        again = [buf.empty_symmetric([T, H], torch.bfloat16) for _ in range(8)]
        assert late_at in [f.data_ptr() for f in again]
    finally:
        vc.destroy()


def test_layout_scratch_outgrown_while_another_stream_uses_it():
    """Layouts of growing size on the caller's, the delayed communication and a third stream: each call has the scratch to itself, and
    what is allocated in between does not get the outgrown one too early."""
    vc, buf = _buffer()
    try:
        sizes = [2500, 2500, 5000, 9000, 9000, 20000]
        idx = [make_routing(n, E, K, "cuda", seed=6 + i)[0] for i, n in enumerate(sizes)]
        want = [torch.bincount(i.flatten(), minlength=E) for i in idx]
        torch.cuda.synchronize()
        side, got, keep = torch.cuda.Stream(), [], []
        for i, n in enumerate(sizes):
            if i % 3 == 1:
                _delay(buf.comm_stream)
                lay, ev = _layout(buf, idx[i], async_finish=True)
                got.append(lay["num_tokens_per_expert"])
                keep.append(ev)
            else:
                with torch.cuda.stream(side if i % 3 == 2 else torch.cuda.current_stream()):
                    got.append(_layout(buf, idx[i])[0]["num_tokens_per_expert"])
            for stream in (torch.cuda.current_stream(), side, buf.comm_stream):
                with torch.cuda.stream(stream):
                    keep.append([torch.full((m,), 7, dtype=torch.int32, device="cuda") for m in (250, 500, 1000, 2000)])
        torch.cuda.synchronize()
        for g, w in zip(got, want):
            assert torch.equal(g.long(), w)
        for k in keep:
            assert not isinstance(k, list) or all(bool((t == 7).all()) for t in k)
    finally:
        vc.destroy()


def test_fused_layers_of_one_buffer_on_two_streams():
    """Two layers that share a buffer, each on a stream of its own: the count exchanges and dispatches share the buffer's words."""
    from deepep_efa_b200.models.moe import MoEConfig, MoELayer
    vc, buf = _buffer(nvl=512 << 20)
    try:
        layers = [MoELayer(MoEConfig(hidden=512, intermediate=256, num_experts=e, num_topk=k, init_std=0.05), buf, seed=e) for e, k in ((64, 6), (16, 2))]
        tokens = (4000, 700)
        data = []
        for i, (layer, n) in enumerate(zip(layers, tokens)):
            layer.prepare_fp8(native_block_scaling=i == 0)
            idx, w = make_routing(n, layer.cfg.num_experts, layer.cfg.num_topk, "cuda", seed=20 + i, masked_fraction=0.1)
            data.append((make_tokens(n, 512, "cuda", seed=20 + i), idx, w))
        want = [layer.forward_fused(*d).clone() for layer, d in zip(layers, data)]
        streams = [torch.cuda.Stream() for _ in layers]
        torch.cuda.synchronize()
        for _ in range(10):
            got = []
            for _ in range(3):
                for layer, d, stream in zip(layers, data, streams):
                    with torch.cuda.stream(stream):
                        got.append(layer.forward_fused(*d))
            torch.cuda.synchronize()
            buf.check_status(sync=True)
            assert all(torch.equal(g, want[i % 2]) for i, g in enumerate(got))
    finally:
        vc.destroy()


def test_calls_that_alternate_between_streams():
    """Direct calls on two streams and asynchronous ones on the communication stream, the host never waiting in between."""
    vc, buf = _buffer()
    try:
        sets = []
        for i, n in enumerate((300, 4000, 37)):
            idx, w = make_routing(n, E, K, "cuda", seed=30 + i, masked_fraction=0.2)
            x = make_tokens(n, H, "cuda", seed=30 + i)
            want = x.float() * (idx >= 0).any(1, keepdim=True)
            sets.append((x, idx, w, want.to(torch.bfloat16)))
        side = torch.cuda.Stream()
        torch.cuda.synchronize()
        got = []
        for step in range(30):
            x, idx, w, want = sets[step % 3]
            how = dict(async_finish=True) if step % 4 in (1, 2) else {}
            with torch.cuda.stream(side if step % 5 == 3 else torch.cuda.default_stream()):
                lay, ev = _layout(buf, idx, **how)
                ev.current_stream_wait()
                y, _, rw, _, handle, ev = buf.dispatch(x, topk_weights=w, **lay, **how)
                ev.current_stream_wait()
                how = dict(async_finish=True) if step % 4 in (2, 3) else {}
                out, out_w, ev = buf.combine(y, handle, topk_weights=rw, **how)
                ev.current_stream_wait()
                got.append((out, out_w, want, w * (idx >= 0)))
            del lay, handle, y, rw
        torch.cuda.synchronize()
        buf.check_status(sync=True)
        for out, out_w, want, want_w in got:
            assert torch.equal(out, want) and torch.equal(out_w, want_w)
    finally:
        vc.destroy()


@pytest.mark.parametrize("how", ["asynchronous", "own_work"])
def test_symmetric_memory_dropped_while_the_communication_stream_uses_it(how):
    """By an asynchronous call of the library, or by work of the caller who asked for the stream."""
    vc, buf = _buffer(nvl=64 << 20)
    try:
        idx, _ = make_routing(T, E, K, "cuda", seed=40)
        x = make_tokens(T, H, "cuda", seed=40)
        lay, _ = _layout(buf, idx)
        y, _, _, _, handle, _ = buf.dispatch(x, **lay)
        late = buf.empty_symmetric([T, H], torch.bfloat16)
        late.copy_(y)
        want, late_at = buf.combine(late, handle)[0].clone(), late.data_ptr()
        start = torch.cuda.Event()
        side = torch.cuda.Stream()
        torch.cuda.synchronize()
        _delay(side)
        start.record(side)
        if how == "asynchronous":  # (without asking for the stream)
            from deepep_efa_b200 import EventOverlap
            from deepep_efa_b200.utils.event import EventHandle
            handle_of_side = EventHandle(record=False)
            handle_of_side.event = start
            out, _, ev = buf.combine(late, handle, previous_event=EventOverlap(handle_of_side), async_finish=True)
        else:
            out, ev = torch.empty_like(want), None
            buf.comm_stream.wait_event(start)
            with torch.cuda.stream(buf.comm_stream):
                out.copy_(late)
            want = y.clone()
        del late
        if ev is not None:
            ev.extra_tensors = ()
        fresh = [buf.empty_symmetric([T, H], torch.bfloat16).fill_(3.0) for _ in range(4)]
        assert late_at not in [f.data_ptr() for f in fresh]
        torch.cuda.synchronize()
        buf.check_status()
        assert torch.equal(out, want)
    finally:
        vc.destroy()


def test_counts_of_a_call_that_did_not_wait_do_not_reach_the_next_one():
    """A dispatch with num_worst_tokens is still queued when the next dispatch waits on the host for its own, larger counts."""
    vc, buf = _buffer()
    try:
        sets = [(make_tokens(n, H, "cuda", seed=50 + n), make_routing(n, E, K, "cuda", seed=50 + n)[0]) for n in (20, 300)]
        lays = [_layout(buf, idx)[0] for _, idx in sets]
        want = buf.dispatch(sets[1][0], **lays[1])[3]
        torch.cuda.synchronize()
        _delay(torch.cuda.current_stream())
        few = buf.dispatch(sets[0][0], num_worst_tokens=64, **lays[0])
        many = buf.dispatch(sets[1][0], **lays[1])
        torch.cuda.synchronize()
        buf.check_status()
        assert torch.equal(many[0], sets[1][0]) and many[3] == want
        assert torch.equal(few[0][:20], sets[0][0]) and few[3] == []
    finally:
        vc.destroy()


@pytest.mark.parametrize("warm", [False, True])
def test_captured_layout_replayed_after_larger_ones(warm):
    """A captured layout keeps scratch memory of its own, whether the buffer had some before or needs more later."""
    vc, buf = _buffer()
    try:
        small, large = (make_routing(n, E, K, "cuda", seed=n)[0] for n in (5000, 40000))
        want = [torch.bincount(i.flatten(), minlength=E) for i in (small, large)]
        if warm:
            _layout(buf, small)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = _layout(buf, small)[0]["num_tokens_per_expert"]
        for _ in range(3):
            eager = _layout(buf, large)[0]["num_tokens_per_expert"]
            keep = [torch.full((n,), 7, dtype=torch.int32, device="cuda") for n in (512, 1024, 2048, 4096) for _ in range(8)]
            captured.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(captured.long(), want[0]) and torch.equal(eager.long(), want[1])
            assert all(bool((t == 7).all()) for t in keep)
    finally:
        vc.destroy()


@pytest.mark.parametrize("form", ["asynchronous", "allocated_there", "with_event_only"])
def test_inputs_dropped_behind_calls_on_the_communication_stream(form):
    """Inputs that die while the communication stream has yet to read them, results used on the caller's stream, and an event that was never recorded."""
    from deepep_efa_b200 import Buffer
    from deepep_efa_b200.utils.event import EventHandle, EventOverlap
    vc, buf = _buffer()
    try:
        idx, _ = make_routing(T, E, K, "cuda", seed=3, masked_fraction=0.2)
        x, y, bias = (make_tokens(T, H, "cuda", seed=s) for s in (3, 4, 5))
        lay, _ = _layout(buf, idx)
        recv, _, _, _, handle, _ = buf.dispatch(x, **lay)
        y = y[:recv.size(0)].contiguous()
        want = recv.clone(), buf.combine(y, handle, bias=bias)[0].clone()
        how = dict(async_finish=form != "with_event_only", allocate_on_comm_stream=form == "allocated_there")
        for _ in range(3):
            parts = [t.clone() for t in (x, y, bias)]
            torch.cuda.synchronize()
            _delay(buf.comm_stream)
            rows, _, _, _, _, first = buf.dispatch(parts[0], handle=handle, previous_event=Buffer.capture(), **how)
            out, _, second = buf.combine(parts[1], handle, bias=parts[2], previous_event=EventOverlap(EventHandle(record=False)), **how)
            extra = [first.extra_tensors, second.extra_tensors]
            assert (extra == [None, None]) == (form == "with_event_only")
            waits = first.event, second.event  # (without the objects that keep the inputs alive)
            del parts, first, second, extra
            keep = _overwrite([(T, H // 2), (want[0].size(0), H // 2)])
            for event in waits:
                if event is not None:
                    event.current_stream_wait()
            assert torch.equal(rows, want[0]) and torch.equal(out, want[1])
            del rows, out, keep
    finally:
        vc.destroy()


@pytest.mark.parametrize("asynchronous", [False, True])
@pytest.mark.parametrize("entry", ["one", "many"])
def test_results_of_a_combine_behind_an_event(entry, asynchronous):
    """A block that the caller's stream gave up after the event, but has yet to write and read, does not become a result of a combine that waits for the
    event alone."""
    from deepep_efa_b200 import Buffer
    from deepep_efa_b200.buffer import _combine_many
    vc, buf = _buffer()
    try:
        idx, w = make_routing(T, E, K, "cuda", seed=7, masked_fraction=0.2)
        x = make_tokens(T, H, "cuda", seed=7)
        lay, _ = _layout(buf, idx)
        y, _, rw, _, handle, _ = buf.dispatch(x, topk_weights=w, **lay)
        want, want_w = (t.clone() for t in buf.combine(y, handle, topk_weights=rw)[:2])
        fives, kept = torch.full_like(want, 5.0), torch.zeros_like(want)
        sixes, kept_w = torch.full_like(want_w, 6.0), torch.zeros_like(want_w)
        torch.cuda.synchronize()
        how = dict(previous_event=Buffer.capture(), async_finish=asynchronous)
        _delay(torch.cuda.current_stream())
        blocks = torch.empty_like(want), torch.empty_like(want_w)
        for block, value, copy in zip(blocks, (fives, sixes), (kept, kept_w)):
            block.copy_(value)
            copy.copy_(block)
        del blocks, block
        if entry == "one":
            out, out_w, ev = buf.combine(y, handle, topk_weights=rw, **how)
        else:
            out, out_w, ev = _combine_many([buf], [(y, handle, rw, None)], Buffer.get_combine_config(1), how["previous_event"], asynchronous, False)[0]
        ev.current_stream_wait()
        torch.cuda.synchronize()
        buf.check_status()
        assert torch.equal(kept, fives) and torch.equal(kept_w, sixes)
        assert torch.equal(out, want) and torch.equal(out_w, want_w)
    finally:
        vc.destroy()


@pytest.mark.parametrize("asynchronous", [False, True])
def test_ids_of_32_bits_behind_an_event(asynchronous):
    """Written on a third stream and covered by the event, while the caller's stream is busy with something else: they are widened behind the event, not
    behind (or in front of) the caller's work, and may be dropped."""
    from deepep_efa_b200.utils.event import EventHandle, EventOverlap
    vc, buf = _buffer()
    try:
        idx, w = make_routing(T, E, K, "cuda", seed=8, masked_fraction=0.2)
        x = make_tokens(T, H, "cuda", seed=8)
        lay, _ = _layout(buf, idx)
        want = [t.clone() for t in (lay["num_tokens_per_expert"], lay["is_token_in_rank"])]
        y, want_idx, want_w, counts, handle, _ = buf.dispatch(x, topk_weights=w, **lay)
        narrow, side = idx.int(), torch.cuda.Stream()
        for caller_busy in (False, True):
            ids = torch.full_like(narrow, -1)
            torch.cuda.synchronize()
            with torch.cuda.stream(side):
                torch.cuda._sleep(DELAY)
                ids.copy_(narrow)
                written = EventOverlap(EventHandle())
            if caller_busy:
                _delay(torch.cuda.current_stream())
                torch.cuda._sleep(DELAY)
            per_rank, _, per_expert, in_rank, ev = buf.get_dispatch_layout(ids, E, previous_event=written, async_finish=asynchronous)
            ev = ev if asynchronous else written
            got = buf.dispatch(x, num_tokens_per_rank=per_rank, is_token_in_rank=in_rank, num_tokens_per_expert=per_expert, topk_idx=ids, topk_weights=w,
                               previous_event=ev if asynchronous else None, async_finish=asynchronous)
            got_event = buf.dispatch(x, num_tokens_per_rank=per_rank, is_token_in_rank=in_rank, num_tokens_per_expert=per_expert, topk_idx=ids, topk_weights=w,
                                     previous_event=ev, async_finish=asynchronous)
            del ids
            keep = _overwrite([(T, K)])
            for out in (got, got_event):
                out[5].current_stream_wait()
            assert torch.equal(per_expert, want[0]) and torch.equal(in_rank, want[1])
            for out in (got, got_event):
                assert out[3] == counts and torch.equal(out[0], y) and torch.equal(out[1], want_idx) and torch.equal(out[2], want_w)
            del keep
        buf.check_status(sync=True)
    finally:
        vc.destroy()


@pytest.mark.parametrize("ids", [torch.int64, torch.int32])
def test_inputs_dropped_behind_asynchronous_low_latency_calls(ids):
    """Tokens, ids (widened or not), weights and counters that die while the communication stream has yet to use them."""
    import deepep_efa_b200 as ep
    from deepep_efa_b200.parallel.virtual import VirtualCluster
    n, hidden = 64, 1024
    vc = VirtualCluster(1, num_nvl_bytes=64 << 20, num_rdma_bytes=ep.Buffer.get_low_latency_rdma_size_hint(n, hidden, 1, E), timeout_ms=5000)
    try:
        buf = vc.buffers[0]
        idx, w = make_routing(n, E, K, "cuda", seed=9, masked_fraction=0.2)
        x, y = make_tokens(n, hidden, "cuda", seed=9), make_tokens(E * n, hidden, "cuda", seed=10).view(E, n, hidden)

        def step(given, **how):
            x, idx, w, y, seen = given
            recv, count, handle, first, _ = buf.low_latency_dispatch(x, idx, n, E, cumulative_local_expert_recv_stats=seen, use_fp8=False, **how)
            out, second, _ = buf.low_latency_combine(y, idx, w, handle, **how)
            return recv, count, out, (first, second)

        def fresh():
            return [x.clone(), idx.to(ids), w.clone(), y.clone(), torch.zeros(E, dtype=torch.int32, device="cuda")]

        _, _, want, _ = step(fresh())
        for _ in range(3):
            given = fresh()
            torch.cuda.synchronize()
            _delay(buf.comm_stream)
            recv, count, out, events = step(given, async_finish=True)
            del given
            keep = _overwrite([(n, K), (n, 2 * K), (E,), (n, hidden // 2)]) + _overwrite([(E, n, hidden // 2)], copies=2)
            for event in events:
                event.current_stream_wait()
            torch.cuda.synchronize()
            assert torch.equal(out, want) and count.sum() == (idx >= 0).sum()
            assert not any(bool(t.any()) for t in keep)
            del keep, out
        buf.check_status(sync=True)
    finally:
        vc.destroy()
