"""Normal mode of a lone rank: the kernels that take the whole GPU against the general ones, which a caller's own config still selects."""
import pytest
import torch

from helpers import make_routing, make_tokens

pytestmark = pytest.mark.gpu


# fewer tokens than a CTA has warps, hidden sizes below, at and past the pieces of a row (1024 channels when casting, 256 and 128 columns of 16
# bytes otherwise) and not a multiple of them, tokens that nobody selected
@pytest.mark.parametrize("T,H,masked", [(1, 128, 0.0), (3, 896, 0.5), (7, 1024, 0.0), (61, 1152, 0.6), (200, 2048, 0.6), (33, 2176, 0.0), (129, 4224, 0.5),
                                        (64, 8192, 0.0)])
@pytest.mark.parametrize("wire", ["bf16", "fp8", "cast", "cast_pow2"])
def test_lone_rank_matches_general_kernels(T, H, masked, wire):
    from deepep_efa_b200 import Config
    from deepep_efa_b200.parallel.virtual import VirtualCluster
    E, K = 8, 2
    vc = VirtualCluster(1, num_nvl_bytes=64 << 20, timeout_ms=2000)
    try:
        buf = vc.buffers[0]
        idx, w = make_routing(T, E, K, "cuda", seed=T, masked_fraction=masked)
        x = make_tokens(T, H, "cuda", seed=H)
        if wire == "fp8":
            x = (x.to(torch.float8_e4m3fn), torch.rand(T, H // 128, device="cuda"))
        per_rank, _, per_expert, in_rank, _ = buf.get_dispatch_layout(idx, E)
        res = []
        for config in (Config(24), None):
            for worst in (0, T + 5):
                rx, ri, rw, counts, handle, _ = buf.dispatch(
                    x, num_tokens_per_rank=per_rank, is_token_in_rank=in_rank, num_tokens_per_expert=per_expert, topk_idx=idx, topk_weights=w, config=config,
                    quantize_fp8=wire.startswith("cast"), round_scale=wire == "cast_pow2", num_worst_tokens=worst)
                n = int(per_rank.item())
                flat = list(rx) if isinstance(rx, tuple) else [rx]
                out = [t[:n].view(torch.uint8).clone() for t in flat] + [ri.clone() if worst else ri[:n].clone(), rw[:n].clone(), handle[3][:n].clone()]
                if worst:
                    assert (ri[n:] == -1).all()
                    res.append(out)
                    continue
                y = torch.randn(n, H, device="cuda", generator=torch.Generator("cuda").manual_seed(1)).to(torch.bfloat16)
                bias = [make_tokens(T, H, "cuda", seed=s) for s in (5, 6)]
                for b in (None, bias[0], tuple(bias)):
                    for placed in (y, buf.empty_symmetric([n, H], torch.bfloat16).copy_(y)):
                        z, zw, _ = buf.combine(placed, handle, topk_weights=rw, bias=b, config=config)
                        out += [z.clone(), zw.clone()]
                cached = buf.dispatch(x, handle=handle, config=config)[0]
                out += [t.view(torch.uint8).clone() for t in (cached if isinstance(cached, tuple) else (cached,))]
                res.append(out)
        buf.check_status(sync=True)
        for a, b in zip(res[:2], res[2:]):
            assert len(a) == len(b) and all(torch.equal(p, q) for p, q in zip(a, b))
    finally:
        vc.destroy()


@pytest.mark.parametrize("async_finish", [False, True])
def test_named_ranges_and_handle_checks_are_of_the_path_that_runs(monkeypatch, async_finish):
    """With NVTX ranges and the debug checks on, dispatch and combine take the same path as without them."""
    from deepep_efa_b200 import buffer as module
    from deepep_efa_b200.parallel.virtual import VirtualCluster
    from deepep_efa_b200.utils import profiler
    T, H, E, K = 40, 512, 8, 2
    vc = VirtualCluster(1, num_nvl_bytes=64 << 20, timeout_ms=2000)
    try:
        buf, names = vc.buffers[0], []
        idx, w = make_routing(T, E, K, "cuda", seed=1)
        x = make_tokens(T, H, "cuda", seed=2)
        per_rank, _, per_expert, in_rank, _ = buf.get_dispatch_layout(idx, E)
        how = dict(async_finish=async_finish)
        fresh = dict(num_tokens_per_rank=per_rank, is_token_in_rank=in_rank, num_tokens_per_expert=per_expert, topk_idx=idx, topk_weights=w, **how)

        def steps():
            rx, _, rw, _, handle, e0 = buf.dispatch(x, **fresh)
            e0.current_stream_wait()
            again, _, _, _, _, e1 = buf.dispatch(x, handle=handle, **how)
            e1.current_stream_wait()
            out, _, e2 = buf.combine(again, handle, **how)
            e2.current_stream_wait()
            torch.cuda.synchronize()
            return handle, [rx.clone(), again.clone(), out.clone()]

        _, plain = steps()

        def other_path(*args, **kw):
            raise AssertionError("the path of several emulated ranks")

        monkeypatch.setattr(module, "_dispatch_many", other_path)
        monkeypatch.setattr(module, "_combine_many", other_path)
        for m in (module, profiler):
            monkeypatch.setattr(m, "NVTX_ENABLED", True)
        monkeypatch.setattr(module, "_DEBUG_CHECKS", True)
        monkeypatch.setattr(torch.cuda.nvtx, "range_push", names.append)
        monkeypatch.setattr(torch.cuda.nvtx, "range_pop", lambda: None)
        handle, named = steps()
        assert names == ["ep.dispatch", "ep.dispatch", "ep.combine"]
        assert all(torch.equal(a, b) for a, b in zip(plain, named))
        foreign = handle[:3] + (handle[3][:-1],) + handle[4:]  # one row short
        with pytest.raises(AssertionError, match="receive count"):
            buf.dispatch(x, handle=foreign, **how)
        with pytest.raises(AssertionError, match="receive count"):
            buf.combine(x[:T - 1], foreign, **how)
    finally:
        vc.destroy()


@pytest.mark.parametrize("T", [0, 31, 256, 1024, 1025, 1056, 8192, 8193, 8200, 20000])
@pytest.mark.parametrize("masked", [0.0, 0.7])
def test_counts_and_positions_of_a_lone_rank(T, masked):
    """Layout by one CTA, by a cluster and by tickets, and the numbering of the tokens that are sent, with the flags of up to eight tokens per thread and of more."""
    from deepep_efa_b200.parallel.virtual import VirtualCluster
    E, K, H = 72, 6, 128
    vc = VirtualCluster(1, num_nvl_bytes=128 << 20, timeout_ms=5000)
    buf = vc.buffers[0]
    try:
        gen = torch.Generator(device="cuda").manual_seed(T)
        idx = torch.rand(T, E, device="cuda", generator=gen).topk(K, dim=1).indices
        idx[torch.rand(T, device="cuda", generator=gen) < masked] = -1  # tokens that stay at home
        x = torch.randn(T, H, device="cuda", generator=gen).to(torch.bfloat16)
        per_rank, _, per_expert, in_rank, _ = buf.get_dispatch_layout(idx, E)
        sent = (idx >= 0).any(dim=1)
        counts = torch.bincount(idx[idx >= 0], minlength=E)
        assert per_rank.tolist() == [int(sent.sum())] and torch.equal(per_expert.long(), counts) and torch.equal(in_rank[:, 0], sent)
        recv, recv_idx, _, per_expert_list, handle, _ = buf.dispatch(x, num_tokens_per_rank=per_rank, is_token_in_rank=in_rank, num_tokens_per_expert=per_expert,
                                                                     topk_idx=idx, topk_weights=torch.ones(T, K, device="cuda"), expert_alignment=8)
        rpm, cpm, rcpm, src_idx, _, head = handle
        assert per_expert_list == ((counts + 7) // 8 * 8).tolist() and rpm.tolist() == [[int(sent.sum())]]
        position = torch.where(sent, sent.cumsum(0) - 1, -1)
        assert torch.equal(head[:, 0].long(), position) and torch.equal(src_idx.long(), sent.nonzero()[:, 0])
        channels = cpm.size(1)
        ends = [min((c + 1) * -(-T // channels), T) for c in range(channels)]
        assert cpm[0].tolist() == [int(sent[:e].sum()) for e in ends] and torch.equal(cpm, rcpm)
        assert torch.equal(recv, x[sent]) and torch.equal(recv_idx, idx[sent])
    finally:
        vc.destroy()
