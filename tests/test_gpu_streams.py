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
