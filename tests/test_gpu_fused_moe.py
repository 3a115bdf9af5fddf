"""Fused MoE forward on emulated ranks (one GPU): expert-major dispatch placement against a host restatement, and the
whole pipeline (arrival-gated GEMM1, cast, GEMM2 with the scatter epilogue, home-side reduce) against a dense fp32 loop
over all experts and against the unfused FP8 path, which does the same arithmetic."""
import pytest
import torch

from helpers import make_routing, make_tokens

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp(min=1e-12)).item()


def _setup(R, T, H, I, E, K, native, seed=0, masked=0.05):
    from deepep_efa_b200.models.moe import MoEConfig, MoELayer
    from deepep_efa_b200.parallel.virtual import VirtualCluster
    L = E // R
    rows = (R * T * min(K, L) + L * 127 + 127) // 128 * 128
    sym = rows * (H + (H // 128) * 4 + 4) + T * K * H * 2
    vc = VirtualCluster(R, num_nvl_bytes=(8 << 20) + 3 * sym, timeout_ms=3000)
    cfg = MoEConfig(hidden=H, intermediate=I, num_experts=E, num_topk=K, init_std=0.05)
    layers = [MoELayer(cfg, vc.buffers[r], seed=seed) for r in range(R)]
    for l in layers:
        l.prepare_fp8(native_block_scaling=native)
    xs = [make_tokens(T, H, "cuda", seed=seed + 10 + r) for r in range(R)]
    idxs, ws = [], []
    for r in range(R):
        i, w = make_routing(T, E, K, "cuda", seed=seed + 20 + r, masked_fraction=masked)
        idxs.append(i), ws.append(w)
    return vc, layers, xs, idxs, ws


@pytest.mark.parametrize("R,T,H,E,K,native", [(2, 70, 512, 8, 3, False), (4, 33, 1024, 16, 4, True), (1, 200, 512, 4, 2, False)])
def test_expert_major_dispatch_places_rows(R, T, H, E, K, native):
    """After em_notify + em_dispatch every local expert's block holds the quantised rows of (source rank, token order),
    the row-info words name (source rank, selection), group offsets are 128-aligned and the arrival counters equal the
    expected totals."""
    import deepep_efa_b200 as ep
    from deepep_efa_b200.models.moe import UNIT_ROWS
    from deepep_efa_b200.reference import oracle
    vc, layers, xs, idxs, ws = _setup(R, T, H, 256, E, K, native)
    try:
        C = ep._ext.load()
        L = E // R
        rts = [b.runtime for b in vc.buffers]
        wss = [l.fused_workspace(T) for l in layers]
        for rep in range(2):  # the second call reuses every buffer and moves the monotonic counters on
            C.em_notify(rts, [(i, w.recv_x, w.recv_scales_raw, w.recv_info, w.stage, w.my_counts, w.sel_list, w.send_base, w.unit_start,
                               w.m_offsets, w.m_ends, w.peer_bases) for i, w in zip(idxs, wss)], E, UNIT_ROWS)
            dst_rows = [torch.full((T * K,), -1, dtype=torch.int32, device="cuda") for _ in range(R)]
            if rep == 0:   # rows quantised by the dispatch kernel itself
                C.em_dispatch(rts, [(x, w.my_counts, w.sel_list, w.send_base, w.unit_start, w.peer_bases, dr, None, None)
                                    for x, w, dr in zip(xs, wss, dst_rows)], E, K, UNIT_ROWS, native, native, 8)
            else:          # rows quantised once per token beforehand, the dispatch only copies
                pre = [C.per_token_cast_to_fp8(x, native, False) for x in xs]
                C.em_dispatch(rts, [(q, w.my_counts, w.sel_list, w.send_base, w.unit_start, w.peer_bases, dr, None, sc)
                                    for (q, sc), w, dr in zip(pre, wss, dst_rows)], E, K, UNIT_ROWS, native, native, 8)
            torch.cuda.synchronize()
            for b in vc.buffers:
                b.check_status()
            for d in range(R):
                w = wss[d]
                offs, ends = w.m_offsets.tolist(), w.m_ends.tolist()
                assert all(o % 128 == 0 for o in offs)
                assert torch.equal(w.arrived, w.expected)
                info = w.recv_info.cpu()
                rx = w.recv_x.cpu().view(torch.uint8)
                for le in range(L):
                    e = d * L + le
                    row = offs[le]
                    for src in range(R):
                        toks, ks = (idxs[src].cpu() == e).nonzero(as_tuple=True)
                        n = toks.numel()
                        if n == 0:
                            continue
                        q, s = oracle.per_token_cast_to_fp8(xs[src].cpu()[toks], round_scale=native)
                        assert torch.equal(rx[row:row + n], q.view(torch.uint8)), (d, le, src)
                        assert torch.equal(info[row:row + n], (src << 24) | (toks * K + ks).int())
                        assert torch.equal(dst_rows[src].cpu()[(toks * K + ks)], torch.arange(row, row + n, dtype=torch.int32))
                        if not native:
                            assert torch.equal(w.recv_scales.cpu()[row:row + n], s)
                        else:
                            atoms = w.recv_scales.cpu()
                            rr = torch.arange(row, row + n)
                            for kb in (0, H // 128 - 1):
                                got = atoms[rr // 128, kb, (rr % 32) * 16 + ((rr // 32) % 4) * 4]
                                want = ((s[:, kb].contiguous().view(torch.int32) >> 23) & 0xff).to(torch.uint8)
                                assert torch.equal(got, want)
                        row += n
                    assert row == ends[le]
                    if le + 1 < L:
                        assert offs[le + 1] == (ends[le] + 127) // 128 * 128
    finally:
        vc.destroy()


@pytest.mark.parametrize("R,T,H,I,E,K,native", [(2, 150, 512, 256, 8, 3, False), (4, 96, 1024, 256, 16, 4, True), (1, 256, 512, 256, 8, 2, True),
                                                   (1, 1024, 512, 256, 2, 2, True)])
def test_fused_forward_matches_dense_and_unfused(R, T, H, I, E, K, native):
    import deepep_efa_b200 as ep
    from deepep_efa_b200.models.moe import dense_reference, fused_forward_many
    vc, layers, xs, idxs, ws = _setup(R, T, H, I, E, K, native, seed=3)
    try:
        w13_all = torch.cat([l.w13.detach().float() for l in layers])
        w2_all = torch.cat([l.w2.detach().float() for l in layers])
        for rep in range(3):
            outs = fused_forward_many(layers, xs, idxs, ws)
            torch.cuda.synchronize()
            for b in vc.buffers:
                b.check_status(sync=True)
            assert ep._ext.load().gemm_error(0) == 0
            for r in range(R):
                ref = dense_reference(xs[r], idxs[r], ws[r].masked_fill(idxs[r] == -1, 0), w13_all, w2_all)
                assert torch.isfinite(outs[r].float()).all()
                assert _rel(outs[r], ref) < 8e-2, (rep, r, _rel(outs[r], ref))
        if native and R * T * K >= 512 * E:
            # wide tiles: the first GEMM can quantise its own output (e4m3 + scale atoms) instead of a cast pass in between;
            # the arithmetic is the same, so the layer's result must not change by a bit
            from deepep_efa_b200.models import moe as moe_mod
            moe_mod.FUSE_CAST_INTO_GEMM1 = not moe_mod.FUSE_CAST_INTO_GEMM1
            try:
                outs2 = fused_forward_many(layers, xs, idxs, ws)
                torch.cuda.synchronize()
                for b in vc.buffers:
                    b.check_status(sync=True)
                for r in range(R):
                    assert torch.equal(outs[r], outs2[r])
            finally:
                moe_mod.FUSE_CAST_INTO_GEMM1 = not moe_mod.FUSE_CAST_INTO_GEMM1
    finally:
        vc.destroy()


def test_fused_dispatch_overflow_is_reported_not_written():
    """A receive buffer that is too small for the rows that would land in it: the count exchange sees it on every rank,
    no row moves, and the host gets a status instead of a stray store."""
    import deepep_efa_b200 as ep
    from deepep_efa_b200.buffer import EPTimeoutError
    from deepep_efa_b200.models.moe import UNIT_ROWS
    R, T, H, E, K = 2, 64, 512, 4, 2
    vc, layers, xs, idxs, ws = _setup(R, T, H, 256, E, K, False, masked=0.0)
    try:
        C = ep._ext.load()
        rts = [b.runtime for b in vc.buffers]
        wss = [l.fused_workspace(T, capacity_rows=128) for l in layers]  # 2 * 64 * 2 selections need far more than 128 rows
        for w in wss:
            w.recv_x.view(torch.uint8).fill_(7)
        C.em_notify(rts, [(i, w.recv_x, w.recv_scales_raw, w.recv_info, w.stage, w.my_counts, w.sel_list, w.send_base, w.unit_start,
                           w.m_offsets, w.m_ends, w.peer_bases) for i, w in zip(idxs, wss)], E, UNIT_ROWS)
        C.em_dispatch(rts, [(x, w.my_counts, w.sel_list, w.send_base, w.unit_start, w.peer_bases, None, None, None) for x, w in zip(xs, wss)],
                      E, K, UNIT_ROWS, False, False, 4)
        torch.cuda.synchronize()
        with pytest.raises(EPTimeoutError):
            vc.buffers[0].check_status()
        for w in wss:
            assert (w.recv_x.view(torch.uint8) == 7).all() and w.m_offsets.abs().sum().item() == 0
        for b in vc.buffers:
            b.runtime.clear_status()
    finally:
        vc.destroy()


def test_expert_major_dispatch_with_many_experts_per_cta():
    """More experts than a CTA lists in one pass over the ids (two emulated ranks share the SMs)."""
    test_expert_major_dispatch_places_rows(2, 9, 128, 2048, 4, False)


@pytest.mark.parametrize("T,H,E,K,native", [(1, 128, 4, 1, True), (5, 512, 300, 3, False), (77, 4224, 6, 4, True), (130, 7296, 5, 5, False), (40, 7168, 16, 8, True)])
def test_lone_dispatch_places_rows_like_the_general_one(T, H, E, K, native):
    """The dispatch of a lone rank that may use the whole GPU (token by token) against the one with a bounded number of CTAs (expert by expert): rows,
    scales, row words, places and arrival counts; hidden sizes below, at and past a warp's span, fewer and more experts than a CTA has threads."""
    import deepep_efa_b200 as ep
    from deepep_efa_b200.models.moe import UNIT_ROWS
    vc, layers, xs, idxs, ws = _setup(1, T, H, 256, E, K, native)
    try:
        C = ep._ext.load()
        rt, w, idx = vc.buffers[0].runtime, layers[0].fused_workspace(T), idxs[0]
        q, s = C.per_token_cast_to_fp8(xs[0], native, False)
        got = []
        for sms in (7, 148 * 6):
            for t in (w.recv_x.view(torch.uint8), w.recv_scales_raw, w.recv_info):
                t.zero_()
            C.em_notify([rt], [(idx, w.recv_x, w.recv_scales_raw, w.recv_info, w.stage, w.my_counts, w.sel_list, w.send_base, w.unit_start, w.m_offsets,
                                w.m_ends, w.peer_bases)], E, UNIT_ROWS)
            dst = torch.full((T * K,), -1, dtype=torch.int32, device="cuda")
            C.em_dispatch([rt], [(q, w.my_counts, w.sel_list, w.send_base, w.unit_start, w.peer_bases, dst, None, s)], E, K, UNIT_ROWS, native, native, sms)
            torch.cuda.synchronize()
            assert torch.equal(w.arrived, w.expected)
            got.append([t.clone() for t in (w.recv_x.view(torch.uint8), w.recv_scales_raw, w.recv_info, dst)])
        vc.buffers[0].check_status()
        assert all(torch.equal(a, b) for a, b in zip(*got)) and (got[0][3].view(-1) >= 0).sum() == (idx >= 0).sum()
    finally:
        vc.destroy()


@pytest.mark.parametrize("R,T", [(1, 1), (1, 30), (1, 160), (1, 300), (1, 380), (1, 500), (2, 3), (2, 100), (2, 150), (2, 190)])
def test_fused_forward_with_tokens_as_columns(monkeypatch, R, T):
    """0.4 to 188 rows per expert, up to 60 and from 121 on with tokens as columns, alone and with a peer, whose second GEMM takes narrow tiles
    of rows below 64 per expert and wide ones beyond: bit for bit the layer that takes rows."""
    import deepep_efa_b200 as ep
    from deepep_efa_b200.models import moe as moe_mod
    H, I, E, K = 512, 384, 8, 3
    vc, layers, xs, idxs, ws = _setup(R, T, H, I, E, K, True, seed=T)
    # (from 120 rows on only large layers take columns; the kernels do not mind small ones)
    monkeypatch.setattr(moe_mod, "SECOND_WINDOW_MIN_WEIGHT_BYTES", 0)
    monkeypatch.setattr(moe_mod, "SECOND_WINDOW_MIN_HIDDEN", 0)
    calls = []

    class Spy:
        def __getattr__(self, name):
            return getattr(ep._ext.load(), name)

        def grouped_gemm(self, *args, **kw):
            calls.append((args[4], args[12], kw.get("tokens_as_columns", 0)))
            return ep._ext.load().grouped_gemm(*args, **kw)

    monkeypatch.setattr(moe_mod.MoELayer, "_C", staticmethod(lambda: Spy()))
    try:
        def run():
            outs = moe_mod.fused_forward_many(layers, xs, idxs, ws)
            torch.cuda.synchronize()
            for b in vc.buffers:
                b.check_status(sync=True)
            assert ep._ext.load().gemm_error(0) == 0
            return outs

        got = run()
        rows = R * T * K / E
        columns = moe_mod._token_columns(rows, 0, 0)
        assert (columns != 0) == (rows <= 60 or 120 < rows <= 200)
        for swiglu, atoms, given in calls:
            if swiglu:
                assert given == columns
            else:
                assert given == (columns if R == 1 else 0)
                narrow = rows < moe_mod.WIDE_TILE_MIN_ROWS_PER_EXPERT and (R > 1 or not columns)
                assert any(atoms is l._mx[1 if narrow else 3] for l in layers)
        monkeypatch.setattr(moe_mod, "_token_columns", lambda *_: 0)
        for a, b in zip(got, run()):
            assert torch.equal(a, b) and a.any()
        w13_all, w2_all = (torch.cat([getattr(l, n).detach().float() for l in layers]) for n in ("w13", "w2"))
        for r in range(R):
            ref = moe_mod.dense_reference(xs[r], idxs[r], ws[r].masked_fill(idxs[r] == -1, 0), w13_all, w2_all)
            assert _rel(got[r], ref) < 8e-2  # as in the test of the whole pipeline above
    finally:
        vc.destroy()


@pytest.mark.parametrize("R,T", [(1, 9), (2, 40)])
def test_fused_products_say_how_many_rows_come(monkeypatch, R, T):
    """The workspace has room for many more rows than come, and FP8 with fp32 scales chooses its tiles by their number: both products name it."""
    from deepep_efa_b200.models import moe
    E, K, I = 16, 2, 384
    vc, layers, xs, idxs, ws = _setup(R, T, 512, I, E, K, native=False)
    try:
        C, hints = layers[0]._C(), []

        class Recorder:
            def __getattr__(self, name):
                return getattr(C, name)

            def grouped_gemm(self, a, b, *args, **kw):
                hints.append((b.size(0), b.size(1) == 2 * I, kw.get("rows_hint")))
                return C.grouped_gemm(a, b, *args, **kw)

        monkeypatch.setattr(moe.MoELayer, "_C", staticmethod(lambda: Recorder()))
        moe.fused_forward_many(layers, xs, idxs, ws, overlap=False)
        torch.cuda.synchronize()
        assert len(hints) == 2 * R and {swiglu for _, swiglu, _ in hints} == {True, False}
        for groups, _, hint in hints:
            assert hint == T * K * groups // (E // R)
    finally:
        vc.destroy()


@pytest.mark.parametrize("T,H,E,K,native", [(1, 128, 4, 1, True), (77, 4224, 6, 4, True), (130, 7296, 300, 5, False)])
def test_places_are_kept_where_they_are_asked_for(T, H, E, K, native):
    """A lone rank's dispatch with places reads no lists, one without them goes by the lists alone, and nothing is written behind a list with room to spare."""
    import deepep_efa_b200 as ep
    from deepep_efa_b200.models.moe import UNIT_ROWS
    vc, layers, xs, idxs, ws = _setup(1, T, H, 256, E, K, native)
    try:
        C = ep._ext.load()
        rt, w, idx = vc.buffers[0].runtime, layers[0].fused_workspace(T), idxs[0]
        assert w.places.shape == (T * K, 2) and w.sel_list.numel() == E * T
        q, s = C.per_token_cast_to_fp8(xs[0], native, False)
        roomy = torch.full((E * T + 4 * T * K + 8,), 7, dtype=torch.int32, device="cuda")
        got = []
        for places, lists in ((w.places, False), (None, True), (w.places, True)):
            for t in (w.recv_x.view(torch.uint8), w.recv_scales_raw, w.recv_info):
                t.zero_()
            w.places.fill_(-1)
            C.em_notify([rt], [(idx, w.recv_x, w.recv_scales_raw, w.recv_info, w.stage, w.my_counts, roomy, w.send_base, w.unit_start, w.m_offsets, w.m_ends,
                                w.peer_bases, places)], E, UNIT_ROWS)
            assert (w.places[:, 0] >= 0).sum() == (0 if places is None else (idx >= 0).sum())
            if places is None:
                w.places.fill_(-1)  # no row would move by them
            if not lists:
                roomy[:E * T] = 0   # every row would be token 0's by them
            dst = torch.full((T * K,), -1, dtype=torch.int32, device="cuda")
            C.em_dispatch([rt], [(q, w.my_counts, roomy, w.send_base, w.unit_start, w.peer_bases, dst, None, s, places)], E, K, UNIT_ROWS, native, native, 148 * 6)
            torch.cuda.synchronize()
            assert (roomy[E * T:] == 7).all()
            got.append([t.clone() for t in (w.recv_x.view(torch.uint8), w.recv_scales_raw, w.recv_info, dst)])
        vc.buffers[0].check_status()
        for other in got[1:]:
            assert all(torch.equal(a, b) for a, b in zip(got[0], other))
        assert (got[0][3] >= 0).sum() == (idx >= 0).sum()
        for bad in (w.places[:, 0], w.places.view(-1)[1:], w.places.long()):
            with pytest.raises(ValueError):
                C.em_notify([rt], [(idx, w.recv_x, w.recv_scales_raw, w.recv_info, w.stage, w.my_counts, roomy, w.send_base, w.unit_start, w.m_offsets,
                                    w.m_ends, w.peer_bases, bad)], E, UNIT_ROWS)
    finally:
        vc.destroy()


@pytest.mark.parametrize("T,H,masked", [(1, 128, 0.0), (700, 4224, 0.05), (300, 7168, 1.0)])
def test_arrivals_of_a_lone_rank(T, H, masked):
    """The dispatch with places counts no arrivals, so that nothing that waits for them reads early; the next exchange makes up for it, and a dispatch that does
    count finds the words as if all calls had."""
    import deepep_efa_b200 as ep
    from deepep_efa_b200.models.moe import UNIT_ROWS
    E, K = 40, 3
    vc, layers, xs, idxs, ws = _setup(1, T, H, 256, E, K, False, masked=masked)
    try:
        C = ep._ext.load()
        rt, w, idx = vc.buffers[0].runtime, layers[0].fused_workspace(T), idxs[0]
        q, s = C.per_token_cast_to_fp8(xs[0], False, False)
        counts = torch.bincount(idx[idx >= 0], minlength=E)
        due = w.arrived.clone()
        assert torch.equal(due, w.expected)
        for counted in (False, False, True, True, False, True):
            places = None if counted else w.places
            w.recv_x.view(torch.uint8).zero_()
            C.em_notify([rt], [(idx, w.recv_x, w.recv_scales_raw, w.recv_info, w.stage, w.my_counts, w.sel_list, w.send_base, w.unit_start, w.m_offsets,
                                w.m_ends, w.peer_bases, places)], E, UNIT_ROWS)
            assert torch.equal(w.arrived, due) and torch.equal(w.expected, due + counts)
            C.em_dispatch([rt], [(q, w.my_counts, w.sel_list, w.send_base, w.unit_start, w.peer_bases, None, None, s, places)], E, K, UNIT_ROWS, False, False, 148)
            torch.cuda.synchronize()
            assert torch.equal(w.arrived, due + counts if counted else due)
            due += counts
            for e in range(E):
                toks = (idx == e).nonzero()[:, 0]
                row = int(w.m_offsets[e])
                assert torch.equal(w.recv_x[row:row + toks.numel()].view(torch.uint8), q.view(torch.uint8)[toks])
        vc.buffers[0].check_status()
    finally:
        vc.destroy()
