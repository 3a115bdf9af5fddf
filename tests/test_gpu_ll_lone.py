"""Low-latency kernels of a lone rank against the general kernels (which the hook form still runs) and the oracle."""
import pytest
import torch

from helpers import make_routing, make_tokens

pytestmark = pytest.mark.gpu


def _cluster(T, H, E, arena=2 << 20):
    from deepep_efa_b200 import Buffer
    from deepep_efa_b200.parallel.virtual import VirtualCluster
    return VirtualCluster(1, num_nvl_bytes=arena, num_rdma_bytes=Buffer.get_low_latency_rdma_size_hint(T, H, 1, E), timeout_ms=2000)


def _valid(res):
    """Everything the dispatch defines: counts, layout, and the valid rows of data, scales and source tokens."""
    rx, cnt, handle = res[:3]
    parts = [cnt, handle[1]]
    for e, n in enumerate(cnt.tolist()):
        parts.append(handle[0][e, :n])
        parts += [r[e, :n].view(torch.uint8) for r in (rx if isinstance(rx, tuple) else (rx,))]
    return [p.clone() for p in parts]


# one token and one selection; slices of a row (few tokens), whole rows, rows wider than a CTA, long batches, more selections than a group of
# eight, hidden sizes that end inside a slice
@pytest.mark.parametrize("T,H,E,K,masked,sms", [(1, 7168, 256, 8, 0.0, None), (1, 128, 1, 1, 0.0, None), (5, 1152, 60, 6, 0.1, None), (77, 4096, 64, 6, 0.05, None),
                                                 (128, 7168, 16, 8, 0.0, None), (128, 7168, 16, 8, 0.1, 7), (20, 8320, 8, 3, 0.0, None),
                                                 (40, 1024, 64, 32, 0.2, None), (512, 512, 32, 8, 0.0, None), (513, 512, 32, 8, 0.0, None), (33, 512, 8, 2, 1.0, None)])
@pytest.mark.parametrize("wire", ["bf16", "fp8", "fp8_pow2", "fp8_ue8m0"])
def test_lone_rank_matches_general_kernels(T, H, E, K, masked, sms, wire):
    from deepep_efa_b200 import Buffer
    if wire == "fp8_ue8m0" and H % 512:
        pytest.skip("UE8M0 scales come in words of 512 channels")
    vc = _cluster(T, H, E, arena=(2 << 20) + E * T * H * 2)
    Buffer.set_low_latency_num_sms(sms)
    try:
        buf = vc.buffers[0]
        how = dict(use_fp8=wire != "bf16", round_scale=wire in ("fp8_pow2", "fp8_ue8m0"), use_ue8m0=wire == "fp8_ue8m0")
        idx, w = make_routing(T, E, K, "cuda", seed=T + K, masked_fraction=masked)
        x = make_tokens(T, H, "cuda", seed=H)
        stats = [torch.zeros(E, dtype=torch.int32, device="cuda") for _ in range(2)]
        general = vc.low_latency_dispatch([x], [idx], T, E, return_recv_hook=True, cumulative_stats=[stats[0]], **how)[0]
        general[4]()
        want = _valid(general)
        y = torch.randn(E, T, H, device="cuda").to(torch.bfloat16)
        out = vc.low_latency_combine([y], [idx], [w], [general[2]], return_recv_hook=True)[0]
        out[2]()
        want_y = out[0].clone()
        got = vc.low_latency_dispatch([x], [idx], T, E, cumulative_stats=[stats[1]], **how)[0]
        for a, b in zip(want, _valid(got)):
            assert torch.equal(a, b)
        assert torch.equal(stats[0], stats[1])
        sym = buf.empty_symmetric([E, T, H], torch.bfloat16)
        sym.copy_(y)
        order = torch.randperm(K, device="cuda")  # selections in another order than at the dispatch: ordinary tensors allow it
        for _ in range(3):  # behind a finished dispatch, then right behind one that may still run, in either parity
            assert torch.equal(vc.low_latency_combine([y], [idx], [w], [got[2]])[0][0], want_y)
            assert torch.equal(vc.low_latency_combine([sym], [idx], [w], [got[2]])[0][0], want_y)
            turned = idx[:, order].contiguous(), w[:, order].contiguous()
            got = vc.low_latency_dispatch([x], [idx], T, E, **how)[0]
            z = vc.low_latency_combine([y], [turned[0]], [turned[1]], [got[2]])[0][0]
            # K products summed in another order in fp32, then rounded to BF16
            assert (z.float() - want_y.float()).norm() <= 4e-3 * want_y.float().norm()
            got = vc.low_latency_dispatch([x], [idx], T, E, **how)[0]
            assert torch.equal(vc.low_latency_combine([sym], [idx], [w], [got[2]])[0][0], want_y)
            got = vc.low_latency_dispatch([x], [idx], T, E, **how)[0]
        buf.check_status()
    finally:
        Buffer.set_low_latency_num_sms(None)
        vc.destroy()


def test_lone_rank_pairs_back_to_back():
    """Pairs with other data each time, alternately of the lone and of the general kernels, the combine right behind its dispatch and its
    result in memory that the caller gave back after the dispatch."""
    T, H, E, K = 96, 2048, 32, 4
    vc = _cluster(T, H, E, arena=(2 << 20) + E * T * H * 2)
    try:
        sym = vc.buffers[0].empty_symmetric([E, T, H], torch.bfloat16)
        sym.copy_(torch.randn(E, T, H, device="cuda"))
        batches = [(make_tokens(T, H, "cuda", seed=s), *make_routing(T, E, K, "cuda", seed=s, masked_fraction=0.05)) for s in range(6)]
        outs = []
        for i in range(48):
            x, idx, w = batches[i % 6]
            x = x.clone()
            hook = i % 5 == 4
            res = vc.low_latency_dispatch([x], [idx], T, E, return_recv_hook=hook)[0]
            if hook:
                res[4]()
            del x
            outs.append((i % 6, [r.clone() for r in (res[1], res[2][1])] if i % 7 == 0 else None,
                         vc.low_latency_combine([sym], [idx], [w], [res[2]])[0][0]))
        torch.cuda.synchronize()
        vc.buffers[0].check_status()
        first = {}
        for b, meta, y in outs:
            idx, w = batches[b][1:]
            if b not in first:
                want = torch.zeros(T, H, device="cuda")
                rows = {}
                for t, es in enumerate(idx.tolist()):
                    for k, e in enumerate(es):
                        if e >= 0:
                            want[t] += w[t, k] * sym[e, rows.setdefault(e, 0)].float()
                            rows[e] += 1
                assert (y.float() - want).norm() <= 4e-3 * want.norm()
                first[b] = y
            assert torch.equal(y, first[b])
            if meta is not None:
                n = torch.bincount(idx[idx >= 0], minlength=E)
                assert torch.equal(meta[0].long(), n) and torch.equal(meta[1].view(-1), n)
    finally:
        vc.destroy()


def test_lone_rank_that_masks_itself_sends_nothing():
    T, H, E, K = 16, 1024, 8, 4
    vc = _cluster(T, H, E)
    try:
        buf = vc.buffers[0]
        idx, w = make_routing(T, E, K, "cuda", seed=3)
        buf.low_latency_update_mask_buffer(0, True)
        res = vc.low_latency_dispatch([make_tokens(T, H, "cuda")], [idx], T, E)[0]
        assert res[1].sum().item() == 0 and res[2][1].sum().item() == 0
        y = torch.randn(E, T, H, device="cuda").to(torch.bfloat16)
        assert vc.low_latency_combine([y], [idx], [w], [res[2]])[0][0].abs().sum().item() == 0
        buf.check_status()
    finally:
        vc.destroy()


@pytest.mark.parametrize("R,T,H", [(1, 128, 7168), (1, 3, 1024), (2, 40, 4096)])
def test_combine_of_the_rows_just_received(R, T, H):
    """The landing zone itself as the expert outputs, right behind the dispatch that fills it: a BF16 round trip without experts. Every call has
    other data, so a row read before it has landed shows."""
    from deepep_efa_b200 import Buffer
    from deepep_efa_b200.parallel.virtual import VirtualCluster
    E, K = 16, 4
    vc = VirtualCluster(R, num_nvl_bytes=2 << 20, num_rdma_bytes=Buffer.get_low_latency_rdma_size_hint(T, H, R, E), timeout_ms=2000)
    try:
        routing = [make_routing(T, E, K, "cuda", seed=r, masked_fraction=0.05) for r in range(R)]
        idxs, ws = [i for i, _ in routing], [w for _, w in routing]
        share = [w.masked_fill(i == -1, 0).sum(dim=1, keepdim=True) for i, w in routing]
        g = torch.Generator(device="cuda").manual_seed(T)

        def data():
            return [torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16) for _ in range(R)]

        def step(xs, outs=None):
            res = vc.low_latency_dispatch(xs, idxs, T, E, use_fp8=False)
            return [c[0] for c in vc.low_latency_combine([r[0] for r in res], idxs, ws, [r[2] for r in res], outs=outs)]

        def check(xs, outs):
            for x, o, s in zip(xs, outs, share):
                # K products of one BF16 value in fp32, then rounded to BF16
                assert ((o.float() - x.float() * s).norm(dim=1) <= 4e-3 * (x.float() * s).norm(dim=1) + 1e-6).all()

        batches = [data() for _ in range(24)]
        torch.cuda.synchronize()
        results = [step(b) for b in batches]
        torch.cuda.synchronize()
        for b, o in zip(batches, results):
            check(b, o)
        if R == 1:  # both parities from a graph, with other inputs in place before every replay
            ins, outs = [data(), data()], [[torch.empty(T, H, dtype=torch.bfloat16, device="cuda")] for _ in range(2)]
            s = torch.cuda.Stream()
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=s):
                    for x, o in zip(ins, outs):
                        step(x, o)
            torch.cuda.current_stream().wait_stream(s)
            for _ in range(4):
                for x in ins:
                    x[0].copy_(data()[0])
                graph.replay()
                torch.cuda.synchronize()
                for x, o in zip(ins, outs):
                    check(x, o)
        for b in vc.buffers:
            b.check_status()
    finally:
        vc.destroy()


def _sums(y, idx, w):
    """What a combine of y [E, N, H] returns when rows were numbered in token order, in fp32."""
    rows, want = {}, torch.zeros(idx.size(0), y.size(2), device=y.device)
    for t, es in enumerate(idx.tolist()):
        for k, e in enumerate(es):
            if e >= 0:
                want[t] += w[t, k] * y[e, rows.setdefault(e, 0)].float()
                rows[e] += 1
    return want


@pytest.mark.parametrize("memory", ["ordinary", "symmetric"])
def test_combine_behind_a_kernel_that_lets_it_start(memory):
    """The expert outputs are written between dispatch and combine by a kernel that allows its successor's launch before it has waited itself:
    another combine of the same handle, whose result is the first rows of the second one's input."""
    T, H, E, K = 96, 7168, 8, 4
    vc = _cluster(T, H, E, arena=(2 << 20) + E * T * H * 2)
    try:
        buf = vc.buffers[0]
        src = torch.randn(E, T, H, device="cuda").to(torch.bfloat16)
        y = buf.empty_symmetric([E, T, H], torch.bfloat16) if memory == "symmetric" else torch.empty(E, T, H, dtype=torch.bfloat16, device="cuda")
        for i in range(8):
            idx, w = make_routing(T, E, K, "cuda", seed=i, masked_fraction=0.05)
            x = make_tokens(T, H, "cuda", seed=i)
            src.copy_(torch.randn(E, T, H, device="cuda"))
            y.copy_(src)
            torch.cuda.synchronize()
            h = vc.low_latency_dispatch([x], [idx], T, E)[0][2]
            first = vc.low_latency_combine([src], [idx], [w], [h], outs=[y[0]])[0][0]
            second = vc.low_latency_combine([y], [idx], [w], [h])[0][0]
            torch.cuda.synchronize()
            want = _sums(src, idx, w)
            assert (first.float() - want).norm() <= 4e-3 * want.norm()
            want = _sums(torch.cat([first[None], src[1:]]), idx, w)
            assert (second.float() - want).norm() <= 4e-3 * want.norm()
        buf.check_status()
    finally:
        vc.destroy()


def test_combine_with_other_columns_than_the_dispatch():
    """A top-k list that is wider, narrower or longer than the dispatch's, filled up with -1: ordinary tensors allow it."""
    T, H, E, K = 20, 1024, 8, 3
    vc = _cluster(32, H, E)
    try:
        for i in range(4):
            idx, w = make_routing(T, E, K, "cuda", seed=i, masked_fraction=0.1)
            idx[:, 2] = -1
            y = torch.randn(E, 32, H, device="cuda").to(torch.bfloat16)
            h = vc.low_latency_dispatch([make_tokens(T, H, "cuda", seed=i)], [idx], 32, E)[0][2]
            want = vc.low_latency_combine([y], [idx], [w], [h])[0][0]
            none, zero = torch.full((T, 4), -1, device="cuda"), torch.zeros(T, 4, device="cuda")
            order = [3, 0, 5, 4, 1, 6, 2]
            wide = torch.cat([idx, none], 1)[:, order].contiguous(), torch.cat([w, zero], 1)[:, order].contiguous()
            narrow = idx[:, :2].contiguous(), w[:, :2].contiguous()
            long = torch.cat([idx, none[:7, :3]]), torch.cat([w, zero[:7, :3]])
            for got in (vc.low_latency_combine([y], [wide[0]], [wide[1]], [h])[0][0], vc.low_latency_combine([y], [narrow[0]], [narrow[1]], [h])[0][0]):
                assert torch.equal(got, want)  # two products: one order of summation
            got = vc.low_latency_combine([y], [long[0]], [long[1]], [h])[0][0]
            assert torch.equal(got[:T], want) and not got[T:].any()
        vc.buffers[0].check_status(sync=True)
    finally:
        vc.destroy()


def test_combine_in_another_order_ignores_rows_of_earlier_calls():
    """Behind an expert's rows lie those of earlier calls, with their source tokens. Selections in another order than at the dispatch name such
    a row here, once from the very token."""
    T, H, E = 8, 256, 2
    vc = _cluster(T, H, E)
    try:
        x, y = make_tokens(T, H, "cuda"), torch.randn(E, T, H, device="cuda").to(torch.bfloat16)
        everything = torch.tensor([[0, 1]] * T, device="cuda")
        one = torch.tensor([[0, 1 if t == 5 else -1] for t in range(T)], device="cuda")
        w = torch.rand(T, 2, device="cuda") + 0.5
        for _ in range(2):  # both parities
            vc.low_latency_dispatch([x], [everything], T, E)
        for _ in range(2):
            h = vc.low_latency_dispatch([x], [one], T, E)[0][2]
            got = vc.low_latency_combine([y], [one.flip(1).contiguous()], [w.flip(1).contiguous()], [h])[0][0]
            want = _sums(y, one, w)
            assert (got.float() - want).norm() <= 4e-3 * want.norm()
        vc.buffers[0].check_status(sync=True)
    finally:
        vc.destroy()


def test_combine_of_a_selection_that_was_not_dispatched_is_reported():
    """The staged form waits for a row that nobody sends and ends in a status; the rows that are there still come."""
    from deepep_efa_b200 import EPTimeoutError
    T, H, E, K = 12, 512, 8, 2
    vc = _cluster(T, H, E)
    try:
        buf = vc.buffers[0]
        idx, w = make_routing(T, E, K, "cuda", seed=5)
        y = torch.randn(E, T, H, device="cuda").to(torch.bfloat16)
        h = vc.low_latency_dispatch([make_tokens(T, H, "cuda")], [idx], T, E)[0][2]
        want = vc.low_latency_combine([y], [idx], [w], [h])[0][0]
        other = idx.clone()
        other[3, 1] = next(e for e in range(E) if e not in idx[3].tolist())
        got = vc.low_latency_combine([y], [other], [w], [h])[0][0]
        with pytest.raises(EPTimeoutError):
            buf.check_status(sync=True)
        keep = torch.arange(T, device="cuda") != 3
        assert torch.equal(got[keep], want[keep])
        buf.recover()
        buf.check_status(sync=True)
    finally:
        vc.destroy()


@pytest.mark.parametrize("memory", ["ordinary", "symmetric"])
def test_combine_into_its_own_input(memory):
    """The result in the place of expert outputs that other tokens still need."""
    T, H, E, K = 128, 4096, 8, 4
    vc = _cluster(T, H, E, arena=(2 << 20) + E * T * H * 2)
    try:
        buf = vc.buffers[0]
        y = buf.empty_symmetric([E, T, H], torch.bfloat16) if memory == "symmetric" else torch.empty(E, T, H, dtype=torch.bfloat16, device="cuda")
        for i in range(4):
            idx, w = make_routing(T, E, K, "cuda", seed=i)
            y.copy_(torch.randn(E, T, H, device="cuda"))
            h = vc.low_latency_dispatch([make_tokens(T, H, "cuda", seed=i)], [idx], T, E)[0][2]
            want = _sums(y, idx, w)
            vc.low_latency_combine([y], [idx], [w], [h], outs=[y[i]])
            assert (y[i].float() - want).norm() <= 4e-3 * want.norm()
        buf.check_status(sync=True)
    finally:
        vc.destroy()


@pytest.mark.parametrize("symmetric", [False, True])
def test_wait_statistics_of_a_lone_rank(symmetric):
    """A lone rank that asks for the time it waits gets it (for its own signals), and the same results."""
    from deepep_efa_b200 import Buffer
    T, H, E, K = 64, 2048, 16, 4

    class Solo:
        Get_rank, Get_size, allgather = (lambda self: 0), (lambda self: 1), (lambda self, obj: [obj])

    buf = Buffer(None, (2 << 20) + E * T * H * 2, Buffer.get_low_latency_rdma_size_hint(T, H, 1, E), low_latency_mode=True, explicitly_destroy=True, comm=Solo())
    try:
        idx, w = make_routing(T, E, K, "cuda", seed=1, masked_fraction=0.05)
        x, y = make_tokens(T, H, "cuda"), torch.randn(E, T, H, device="cuda").to(torch.bfloat16)
        if symmetric:
            y = buf.empty_symmetric([E, T, H], torch.bfloat16).copy_(y)
        h = buf.low_latency_dispatch(x, idx, T, E)[2]
        want = buf.low_latency_combine(y, idx, w, h)[0]
        waits = [torch.zeros(1, dtype=torch.int64, device="cuda") for _ in range(2)]
        before = [0, 0]
        for _ in range(3):
            recv, _, h, _, _ = buf.low_latency_dispatch(x, idx, T, E, dispatch_wait_recv_cost_stats=waits[0])
            assert torch.equal(buf.low_latency_combine(y, idx, w, h, combine_wait_recv_cost_stats=waits[1])[0], want)
            now = [t.item() for t in waits]
            assert all(n > b for n, b in zip(now, before))
            before = now
        buf.check_status(sync=True)
    finally:
        buf.destroy()


def test_pull_combine_stores_behind_its_dispatch():
    """The general kernels right behind each other, more tokens than SMs, and a result in the block that held the dispatch's input: every row
    still leaves as it was."""
    from deepep_efa_b200 import Buffer
    T, H, E, K = 400, 2048, 32, 4

    class Solo:
        Get_rank, Get_size, allgather = (lambda self: 0), (lambda self: 1), (lambda self, obj: [obj])

    buf = Buffer(None, (2 << 20) + E * T * H * 2, Buffer.get_low_latency_rdma_size_hint(T, H, 1, E), low_latency_mode=True, explicitly_destroy=True, comm=Solo())
    try:
        y = buf.empty_symmetric([E, T, H], torch.bfloat16)
        y.copy_(torch.randn(E, T, H, device="cuda"))
        idx, w = make_routing(T, E, K, "cuda", seed=2)
        want, waits = _sums(y, idx, w), torch.zeros(1, dtype=torch.int64, device="cuda")
        data = make_tokens(T, H, "cuda")
        for i in range(6):
            x = data.roll(i, 0)
            torch.cuda.synchronize()
            recv, _, h, _, _ = buf.low_latency_dispatch(x, idx, T, E, use_fp8=False, dispatch_wait_recv_cost_stats=waits)
            del x
            out = buf.low_latency_combine(y, idx, w, h, combine_wait_recv_cost_stats=waits)[0]
            rows, x = {}, data.roll(i, 0)
            at = torch.tensor([[rows.setdefault(e, []).append(t) or len(rows[e]) - 1 for e in es] for t, es in enumerate(idx.tolist())], device="cuda")
            assert torch.equal(recv[idx.view(-1), at.view(-1)].view(T, K, H), x[:, None].expand(T, K, H))
            assert (out.float() - want).norm() <= 4e-3 * want.norm()
        buf.check_status(sync=True)
    finally:
        buf.destroy()


def test_phase_stamps_of_a_lone_rank():
    T, H, E, K = 32, 2048, 16, 4
    vc = _cluster(T, H, E, arena=(2 << 20) + E * T * H * 2)
    try:
        buf = vc.buffers[0]
        idx, w = make_routing(T, E, K, "cuda", seed=2)
        y = buf.empty_symmetric([E, T, H], torch.bfloat16)
        buf.runtime.enable_trace(True)
        h = vc.low_latency_dispatch([make_tokens(T, H, "cuda")], [idx], T, E)[0][2]
        vc.low_latency_combine([y], [idx], [w], [h])
        torch.cuda.synchronize()
        trace = buf.runtime.read_trace()
        buf.runtime.enable_trace(False)
        # the two low-latency families, first and last CTA of each: the phases that a kernel without signalling has, in order
        for slot, phases in ((8, (0, 3, 4, 6)), (9, (0, 4, 6)), (10, (0, 4, 5, 6)), (11, (0, 4, 5, 6))):
            at = [trace[slot * 16 + p] for p in phases]
            assert all(at) and at == sorted(at)
    finally:
        vc.destroy()


# both sides of the lines between the two dispatch kernels: the longest lists, narrow rows, a bounded number of SMs, 32 selections per token
@pytest.mark.parametrize("T,H,E,K,masked,sms", [(512, 2048, 32, 8, 0.0, None), (513, 2048, 32, 8, 0.1, None), (119, 512, 32, 8, 0.1, None), (192, 512, 32, 8, 0.0, None),
                                                 (4, 1024, 64, 32, 0.2, None), (30, 2048, 64, 32, 0.2, None), (128, 2048, 16, 8, 0.1, 7), (129, 2048, 16, 8, 0.0, 7)])
@pytest.mark.parametrize("wire", ["bf16", "fp8"])
def test_lone_rank_around_the_lines_of_its_dispatch(T, H, E, K, masked, sms, wire):
    test_lone_rank_matches_general_kernels(T, H, E, K, masked, sms, wire)


# rows of more than 512 columns on few SMs: both sides of the line between the two combine kernels, and the widest rows that have one side
@pytest.mark.parametrize("T,H,sms", [(14, 4224, 7), (15, 4224, 7), (40, 4096, 7), (9, 7168, 4)])
def test_lone_rank_around_the_lines_of_its_combine(T, H, sms):
    test_lone_rank_matches_general_kernels(T, H, 16, 4, 0.1, sms, "fp8")
