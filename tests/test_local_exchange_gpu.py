"""The one-rank kernels of the low-latency calls (csrc/lowlat.cu, ll_local_*) and of the un-fused exchange (csrc/local.cu),
against the window kernels that several ranks use (a buffer with a rank mask takes them on one rank too) and against
plain indexing."""
import pytest
import torch

import teramoe_b200 as tm

pytestmark = pytest.mark.gpu


def _routing(T, E, K, seed, dtype=torch.int64, drop=0.2):
    g = torch.Generator().manual_seed(seed)
    idx = torch.stack([torch.randperm(E, generator=g)[:K] for _ in range(T)]) if T else torch.zeros(0, K, dtype=torch.int64)
    gone = torch.rand(T, K, generator=g) < drop
    if T > 2:
        gone[2] = True                      # a token that goes nowhere
    idx = idx.masked_fill(gone, -1)
    w = torch.rand(T, K, generator=g)
    return idx.to(dtype).cuda(), w.cuda()


# one token; a token per block; fewer tokens than blocks wanted; more; hidden sizes of 1, 2 and 28 channel steps; top-k of 1, 8, 9 and 32
@pytest.mark.parametrize("T,H,E,K,M", [(1, 256, 4, 1, 1), (0, 512, 4, 2, 8), (3, 512, 8, 8, 4), (77, 7168, 32, 8, 128), (300, 1024, 40, 9, 300),
                                       (40, 2560, 64, 32, 64)])
@pytest.mark.parametrize("wire", ["bf16", "fp8", "pow2", "ue8m0"])
def test_low_latency_local_kernels_match_window_kernels(T, H, E, K, M, wire):
    if wire == "ue8m0" and H % 512:
        pytest.skip("UE8M0 scales are packed four groups to a word")
    idx, w = _routing(T, E, K, seed=T + K, dtype=torch.int32 if K == 9 else torch.int64)
    x = (torch.randn(T, H, generator=torch.Generator().manual_seed(T)) * 0.3).to(torch.bfloat16).cuda()
    y = (torch.randn(E, M, H, generator=torch.Generator().manual_seed(H)) * 0.2).to(torch.bfloat16).cuda()
    y[:, :, :128] *= 8.0                    # groups that LogFMT leaves as they are
    got = []
    for shrink in (False, True):            # local kernels, window kernels
        buf = tm.Buffer(None, 0, low_latency_mode=True, explicitly_destroy=True, enable_shrink=shrink)
        stats = torch.zeros(E, dtype=torch.int32, device="cuda")
        recv, count, handle, _, hook = buf.low_latency_dispatch(x, idx, M, E, cumulative_local_expert_recv_stats=stats, use_fp8=wire != "bf16",
                                                                round_scale=wire in ("pow2", "ue8m0"), use_ue8m0=wire == "ue8m0",
                                                                return_recv_hook=True)
        hook()
        assert (handle.entry_row is None) == shrink
        rows, scales = recv if isinstance(recv, tuple) else (recv, None)
        valid = torch.arange(M, device="cuda").view(1, -1) < count.view(-1, 1)
        outs = [count, stats, handle.layout_range, handle.src_info[valid], rows.view(torch.uint8)[valid]]
        if scales is not None:
            outs.append(scales[valid])
        for logfmt in (False, True):
            outs.append(buf.low_latency_combine(y, idx, w, handle, use_logfmt=logfmt)[0])
        # routing with entries removed: their rows are left out
        fewer = idx.masked_fill(torch.arange(K, device="cuda").view(1, -1) % 3 == 1, -1)
        outs.append(buf.low_latency_combine(y, fewer, w, handle)[0])
        torch.cuda.synchronize()
        buf.check_status()
        got.append(outs)
        buf.destroy()
    for i, (a, b) in enumerate(zip(*got)):
        assert torch.equal(a, b), f"output {i} differs"


# top-k of 1 to 4: a block takes 8, 4 or 2 channel steps of 256; nine and ten of them leave a short last block behind full ones
@pytest.mark.parametrize("T,H,E,K,M", [(5, 2304, 4, 1, 8), (6, 2304, 8, 2, 8), (7, 2560, 8, 3, 8), (77, 2304, 16, 4, 128), (3, 256, 8, 4, 4)])
def test_logfmt_combine_of_few_entries_matches_window_kernels(T, H, E, K, M):
    idx, w = _routing(T, E, K, seed=T)
    x = torch.zeros(T, H, dtype=torch.bfloat16, device="cuda")
    y = (torch.randn(E, M, H, generator=torch.Generator().manual_seed(H)) * 0.2).to(torch.bfloat16).cuda()
    y[:, :, :128] *= 8.0                    # groups that LogFMT leaves as they are
    got = []
    for shrink in (False, True):            # local kernels, window kernels
        buf = tm.Buffer(None, 0, low_latency_mode=True, explicitly_destroy=True, enable_shrink=shrink)
        handle = buf.low_latency_dispatch(x, idx, M, E, use_fp8=False)[2]
        assert (handle.entry_row is None) == shrink
        got.append(buf.low_latency_combine(y, idx, w, handle, use_logfmt=True)[0].clone())
        buf.check_status()
        buf.destroy()
    assert torch.equal(*got) and bool(got[0].any())


# chunks of 128 tokens: one, a full one, one more token, several; rows of 2 KB segments: a short one, several, odd byte counts (fp8 scales)
@pytest.mark.parametrize("T,H,E,K", [(0, 256, 4, 2), (1, 128, 4, 1), (128, 1024, 8, 4), (129, 1032, 300, 8), (1003, 7168, 32, 8), (1024, 128, 40, 8), (1025, 128, 40, 8),
                                      (5000, 256, 40, 32)])
@pytest.mark.parametrize("fp8", [False, True])
def test_unfused_exchange_matches_plain_indexing(T, H, E, K, fp8):
    idx, w = _routing(T, E, K, seed=T + H, dtype=torch.int32 if T == 1003 else torch.int64)
    g = torch.Generator().manual_seed(1)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).cuda()
    payload = (x.to(torch.float8_e4m3fn), torch.randn(T, max(1, H // 128), generator=g).cuda()) if fp8 else x
    parts = payload if fp8 else (x,)
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    valid = idx >= 0
    goes = valid.any(1)
    n = int(goes.sum())
    per_rank, _, per_expert, in_rank, _ = buf.get_dispatch_layout(idx, E)
    want_counts = torch.bincount(idx[valid].long(), minlength=E)
    assert per_rank.tolist() == [n] and torch.equal(per_expert.long(), want_counts) and torch.equal(in_rank[:, 0], goes)
    recv, recv_idx, recv_w, counts, handle, _ = buf.deepep_dispatch(payload, topk_idx=idx, topk_weights=w, num_tokens_per_expert=per_expert,
                                                                    expert_alignment=16)
    assert counts == ((want_counts + 15) // 16 * 16).tolist() and recv_idx.dtype == idx.dtype
    assert torch.equal(recv_idx, idx[goes]) and torch.equal(recv_w, torch.where(valid, w, torch.zeros_like(w))[goes])
    for a, b in zip(recv if fp8 else (recv,), parts):
        assert a.dtype == b.dtype and torch.equal(a.contiguous().view(torch.uint8), b[goes].contiguous().view(torch.uint8))
    again = buf.deepep_dispatch(payload, handle=handle)[0]
    for a, b in zip(again if fp8 else (again,), recv if fp8 else (recv,)):
        assert torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8))
    y = torch.randn(n, H, generator=g).to(torch.bfloat16).cuda()
    out, cw, _ = buf.deepep_combine(y, handle, topk_weights=recv_w)
    want = torch.zeros(T, H, dtype=torch.bfloat16, device="cuda")
    want[goes] = y
    assert torch.equal(out, want) and torch.equal(cw, torch.where(valid, w, torch.zeros_like(w)))
    # fixed-shape outputs: rows past the received count are "nothing", and no host wait happens before the combine asks
    worst = T + 5
    recv, recv_idx, recv_w, counts, fixed, ev = buf.deepep_dispatch(payload, topk_idx=idx, topk_weights=w, num_tokens_per_expert=per_expert,
                                                                    num_worst_tokens=worst, async_finish=True)
    ev.current_stream_wait()
    assert counts == [] and fixed.rows == -1 and recv_idx.shape == (worst, K)
    assert torch.equal(recv_idx[:n], idx[goes]) and bool((recv_idx[n:] == -1).all()) and bool((recv_w[n:] == 0).all())
    for a, b in zip(recv if fp8 else (recv,), parts):
        a = a.view(torch.uint8)
        assert a.shape[0] == worst and torch.equal(a[:n], b[goes].contiguous().view(torch.uint8)) and not bool(a[n:].any())
    if n:
        with pytest.raises(ValueError, match="expected"):
            buf.deepep_combine(y[:-1], fixed)
    buf.destroy()


# one block | a cluster of eight, of which the last have nothing, a chunk each, several at a time and a short last one, all that they take | one block per chunk
@pytest.mark.parametrize("T,E,K", [(1024, 5, 2), (1025, 5, 2), (1153, 300, 8), (9001, 2500, 2), (16384, 33, 8), (16385, 33, 8)])
def test_layout_of_many_tokens(T, E, K):
    """Counts, ranks and the rows' order, on the device and as the host reads them; tokens without an expert in every chunk, and a chunk of them."""
    idx, w = _routing(T, E, K, seed=T, dtype=torch.int32 if T % 2 else torch.int64)
    idx[130:300] = -1
    valid = idx >= 0
    goes = valid.any(1)
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    x = torch.arange(T, device="cuda").view(T, 1).expand(T, 4).to(torch.int16).contiguous().view(torch.bfloat16)
    for _ in range(2):
        per_rank, _, per_expert, in_rank, _ = buf.get_dispatch_layout(idx, E)
        want = torch.bincount(idx[valid].long(), minlength=E)
        assert per_rank.tolist() == [int(goes.sum())] and torch.equal(per_expert.long(), want) and torch.equal(in_rank[:, 0], goes)
        recv, recv_idx, _, counts, _, _ = buf.deepep_dispatch(x, topk_idx=idx, topk_weights=w, num_tokens_per_expert=per_expert)
        assert counts == want.tolist() and torch.equal(recv.view(torch.int16), x[goes].view(torch.int16)) and torch.equal(recv_idx, idx[goes])
    buf.destroy()


@pytest.mark.parametrize("T,E,K,M", [(5, 33, 3, 7), (1, 2, 1, 1), (0, 40, 2, 4)])
def test_results_of_a_call_do_not_overlap_and_start_as_allocations_do(T, E, K, M):
    """They lie in one block: every one on a boundary of its own, and writing one leaves the others alone."""
    idx, w = _routing(T, E, K, seed=3, dtype=torch.int64)
    buf = tm.Buffer(None, tm.Buffer.get_low_latency_rdma_size_hint(M, 512, 1, E), low_latency_mode=True, explicitly_destroy=True)
    x = torch.randn(T, 512, device="cuda").to(torch.bfloat16)
    (_, scales), count, handle, _, _ = buf.low_latency_dispatch(x, idx, M, E)
    assert scales.shape == (E, M, 4) and scales.stride() == (4 * M, 1, M)
    per_rank, _, per_expert, in_rank, _ = buf.get_dispatch_layout(idx, E)
    for block in ((handle.layout_range, count, handle.src_info, handle.entry_row), (per_expert, in_rank)):
        block = [t for t in block if t.numel()]
        assert all(t.data_ptr() % 512 == 0 and t.is_contiguous() for t in block)
        for t in block:
            before = [o.clone() for o in block if o is not t]
            t.fill_(1)
            assert all(torch.equal(o, b) for o, b in zip([o for o in block if o is not t], before))
    buf.destroy()


def test_what_a_program_keeps_of_a_call_has_memory_of_its_own():
    """The received counts and the ranks of the tokens hold no other result's memory, and taking more does not reach into one."""
    T, E, K, M = 200, 16, 4, 256
    idx, w = _routing(T, E, K, seed=3, dtype=torch.int64)
    buf = tm.Buffer(None, tm.Buffer.get_low_latency_rdma_size_hint(M, 512, 1, E), low_latency_mode=True, explicitly_destroy=True)
    x = torch.randn(T, 512, device="cuda").to(torch.bfloat16)
    _, count, handle, _, _ = buf.low_latency_dispatch(x, idx, M, E)
    per_rank, _, per_expert, in_rank, _ = buf.get_dispatch_layout(idx, E)
    others = [handle.layout_range, handle.src_info, handle.entry_row, per_rank, per_expert]
    before = [t.clone() for t in others]
    for t in (count, in_rank):
        assert t.untyped_storage().nbytes() == t.numel() * t.element_size()
        t.resize_(1 << 16).fill_(1)
    assert all(torch.equal(t, b) for t, b in zip(others, before))
    buf.destroy()


def _stall(stream, ms=40):
    with torch.cuda.stream(stream):
        torch.cuda._sleep(int(ms * 1.5e6))             # cycles


@pytest.mark.parametrize("call", ["combine", "repeat", "low latency"])
def test_a_handle_of_the_communication_stream_is_waited_for(call):
    """The dispatch runs on the communication stream, behind other work there; the next call on its handle runs on the caller's
    stream and needs nothing else of the dispatch, so nobody has waited for its event."""
    T, H, E, K, M = (8192, 7168, 32, 8, 0) if call != "low latency" else (64, 512, 8, 4, 64)
    idx, w = _routing(T, E, K, seed=5)
    goes = (idx >= 0).any(1)
    buf = tm.Buffer(None, 0, low_latency_mode=True, explicitly_destroy=True)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    if call == "low latency":
        y = torch.randn(E, M, H, device="cuda").to(torch.bfloat16)
        plain = buf.low_latency_dispatch(x, idx, M, E, use_fp8=False)[2]
        want = buf.low_latency_combine(y, idx, w, plain)[0].clone()
    torch.cuda.synchronize()
    _stall(buf.get_comm_stream())
    if call == "low latency":
        handle = buf.low_latency_dispatch(x, idx, M, E, use_fp8=False, async_finish=True)[2]
        got = buf.low_latency_combine(y, idx, w, handle)[0]
    else:
        handle = buf.deepep_dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E, async_finish=True)[4]
        if call == "repeat":
            got, want = buf.deepep_dispatch(x, handle=handle)[0], x[goes]
        else:
            want = torch.where(goes[:, None], x, torch.zeros_like(x))
            got = buf.deepep_combine(x[goes], handle)[0]
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    buf.destroy()


@pytest.mark.parametrize("worst", [0, 1009])
def test_a_handle_of_the_callers_stream_is_waited_for(worst):
    """The other way round: a plain dispatch on a stalled stream, then asynchronous calls behind an event that says nothing of it."""
    T, H, E, K = 1000, 512, 8, 4
    idx, w = _routing(T, E, K, seed=15)
    goes = (idx >= 0).any(1)
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    rows, before = x[goes].contiguous(), buf.capture()
    torch.cuda.synchronize()
    _stall(torch.cuda.current_stream())
    handle = buf.deepep_dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E, num_worst_tokens=worst)[4]
    again = buf.deepep_dispatch(x, handle=handle, previous_event=before, async_finish=True)[0]
    out = buf.deepep_combine(rows, handle, previous_event=before, async_finish=True)[0]
    torch.cuda.synchronize()
    assert torch.equal(again, rows) and torch.equal(out, torch.where(goes[:, None], x, torch.zeros_like(x)))
    buf.destroy()


@pytest.mark.parametrize("call", ["combine", "repeat", "low latency"])
def test_the_tables_of_a_dropped_handle_outlive_the_calls_on_them(call):
    """The handle goes while the call that uses it still waits on the communication stream.  Memory of its size is asked for at once
    and filled with zeros, which are valid rows."""
    T, H, E, K, M = 1000, 512, 8, 4, 1000
    idx, w = _routing(T, E, K, seed=6)
    goes = (idx >= 0).any(1)
    buf = tm.Buffer(None, 0, low_latency_mode=True, explicitly_destroy=True)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    if call == "low latency":
        y = torch.randn(E, M, H, device="cuda").to(torch.bfloat16)
        handle = buf.low_latency_dispatch(x, idx, M, E, use_fp8=False)[2]
        want, n = buf.low_latency_combine(y, idx, w, handle)[0].clone(), T * K
    else:
        y = x[goes].contiguous()
        handle, n = buf.deepep_dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E)[4], T
        want = y if call == "repeat" else torch.where(goes[:, None], x, torch.zeros_like(x))
    torch.cuda.synchronize()
    _stall(buf.get_comm_stream())
    if call == "low latency":
        got = buf.low_latency_combine(y, idx, w, handle, async_finish=True)[0]
    elif call == "repeat":
        got = buf.deepep_dispatch(x, handle=handle, async_finish=True)[0]
    else:
        got = buf.deepep_combine(y, handle, async_finish=True)[0]
    del handle
    reuse = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(8)]
    torch.cuda.synchronize()
    assert torch.equal(got, want) and len(reuse) == 8
    buf.destroy()


def test_a_fixed_shape_handle_counts_its_rows_on_the_stream_of_its_dispatch():
    """dispatch on the stalled communication stream, then a repeat behind its event and a combine of the repeated rows"""
    T, H, E, K = 1000, 512, 8, 4
    idx, w = _routing(T, E, K, seed=7)
    goes = (idx >= 0).any(1)
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    torch.cuda.synchronize()
    _stall(buf.get_comm_stream())
    *_, counts, handle, ev = buf.deepep_dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E, num_worst_tokens=T + 9, async_finish=True)
    assert counts == [] and handle.rows == -1
    *_, ev = got = buf.deepep_dispatch(x, handle=handle, previous_event=ev, async_finish=True)
    ev.current_stream_wait()
    assert torch.equal(got[0], x[goes]) and handle.rows == int(goes.sum())
    assert torch.equal(buf.deepep_combine(got[0], handle)[0], torch.where(goes[:, None], x, torch.zeros_like(x)))
    buf.destroy()


def test_the_rows_of_a_fixed_shape_handle_wait_for_nothing_behind_them():
    T, H, E, K = 300, 512, 8, 4
    idx, w = _routing(T, E, K, seed=8)
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    handle = buf.deepep_dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E, num_worst_tokens=T)[4]
    _stall(torch.cuda.current_stream(), 300)
    behind = torch.cuda.Event()
    behind.record()
    rows = handle.num_rows()
    assert not behind.query()
    assert rows == int((idx >= 0).any(1).sum())
    buf.destroy()


def test_a_fixed_shape_dispatch_in_a_graph_counts_the_rows_of_the_last_replay():
    T, H, E, K = 300, 512, 8, 4
    idx, w = _routing(T, E, K, seed=9)
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    dispatch = lambda: buf.deepep_dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E, num_worst_tokens=T)
    dispatch()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        recv, *_, handle, _ = dispatch()
    for _ in range(2):
        graph.replay()
        goes = (idx >= 0).any(1)
        n = int(goes.sum())
        assert handle.num_rows() == n and torch.equal(recv[:n], x[goes])
        idx[: T // 2] = -1
    buf.destroy()


def test_combine_takes_weights_of_the_received_rows_only():
    """As on the several-rank path, more rows and columns than were sent are accepted and left out; fewer, a vector or host memory are not."""
    T, H, E, K = 300, 512, 8, 4
    idx, w = _routing(T, E, K, seed=10)
    valid = idx >= 0
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    recv, _, recv_w, _, handle, _ = buf.deepep_dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E)
    n = recv.shape[0]
    want = torch.where(valid, w, torch.zeros_like(w))
    wide = torch.full((n + 3, K + 2), 7.0, device="cuda")
    wide[:n, :K] = recv_w
    for good in (recv_w, wide, recv_w.double(), recv_w.t().contiguous().t()):
        assert torch.equal(buf.deepep_combine(recv, handle, topk_weights=good)[1], want)
    for bad in (recv_w[:-1], recv_w[:, :-1], recv_w.reshape(-1), recv_w.cpu()):
        with pytest.raises(RuntimeError, match="topk_weights"):
            buf.deepep_combine(recv, handle, topk_weights=bad)
    for bad in (recv[:-1], recv.float(), recv.reshape(-1)):
        with pytest.raises((ValueError, RuntimeError)):
            buf.deepep_combine(bad, handle)
    buf.destroy()


def test_expert_alignment_of_any_value():
    """What Python's integer arithmetic gives, on which the several-rank path relies: zero raises."""
    T, H, E, K = 100, 256, 8, 4
    idx, w = _routing(T, E, K, seed=11)
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    sent = torch.bincount(idx[idx >= 0], minlength=E).tolist()
    dispatch = lambda a, **kw: buf.deepep_dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E, expert_alignment=a, **kw)[3]
    for a in (1, 7, 128, -4):
        assert dispatch(a) == [(c + a - 1) // a * a for c in sent]
    with pytest.raises(ZeroDivisionError):
        dispatch(0)
    assert dispatch(0, num_worst_tokens=T) == []
    buf.destroy()


def test_dispatch_refuses_what_the_several_rank_path_refuses():
    T, H, E, K = 20, 256, 8, 2
    idx, w = _routing(T, E, K, seed=12)
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    handle = buf.deepep_dispatch(x, topk_idx=idx, topk_weights=w, num_experts=8189)[4]
    for payload in ((x,), (x, x, x)):
        with pytest.raises(ValueError):
            buf.deepep_dispatch(payload, topk_idx=idx, topk_weights=w, num_experts=E)
        with pytest.raises(ValueError):
            buf.deepep_dispatch(payload, handle=handle)
    with pytest.raises(ValueError, match="too many experts"):
        buf.deepep_dispatch(x, topk_idx=idx, topk_weights=w, num_experts=8190)
    buf.destroy()


def test_wait_statistics_are_checked_and_nothing_is_added():
    T, H, E, K = 20, 256, 8, 2
    idx, w = _routing(T, E, K, seed=13)
    buf = tm.Buffer(None, 0, low_latency_mode=True, explicitly_destroy=True)
    x, y = torch.randn(T, H, device="cuda").to(torch.bfloat16), torch.randn(E, T, H, device="cuda").to(torch.bfloat16)
    stats = torch.full((1,), 5, dtype=torch.int64, device="cuda")
    dispatch = lambda t: buf.low_latency_dispatch(x, idx, T, E, dispatch_wait_recv_cost_stats=t)[2]
    handle = dispatch(stats)
    combine = lambda t: buf.low_latency_combine(y, idx, w, handle, combine_wait_recv_cost_stats=t)
    combine(stats)
    assert stats.tolist() == [5]
    for bad in (stats.cpu(), stats.int(), torch.zeros(4, dtype=torch.int64, device="cuda")[::2]):
        for call in (dispatch, combine):
            with pytest.raises(RuntimeError, match="wait_stats"):
                call(bad)
    buf.destroy()


def test_a_backward_pass_of_the_layer_leaves_the_low_latency_windows_to_be_laid_out_again():
    """The windows of a buffer with a rank mask share the arena with the layer: their flags are cleared behind a backward pass too."""
    T, H, E, K, M = 256, 512, 4, 2, 8
    idx, w = _routing(T, E, K, seed=14, drop=0.0)
    buf = tm.Buffer(None, 0, low_latency_mode=True, explicitly_destroy=True, enable_shrink=True)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16).requires_grad_(True)
    Wg, Wd = (torch.randn(E, n, k, device="cuda").to(torch.bfloat16) * 0.02 for n, k in ((256, H), (H, 128)))
    out = buf.teramoe_autograd(x, idx, w, Wg, Wd, E)
    low = lambda: buf.low_latency_dispatch(x.detach()[:M, :256].contiguous(), idx[:M].contiguous(), M, E, use_fp8=False)
    low()
    out.backward(torch.ones_like(out))
    geom = buf._ll_prepare(M, 256, E, False, False, False, False)
    for off, n in ((geom[10], E * 8), (geom[12], E * 8)):
        assert not bool(buf._world.data.view(off, [n // 8], torch.int64).any())
    _, count, *_ = low()
    sent = idx[:M].flatten().long()
    assert torch.equal(count.long(), torch.bincount(sent[sent >= 0], minlength=E))
    buf.check_status()
    buf.destroy()


def test_rows_off_a_16_byte_boundary():
    """Contiguous tensors may start anywhere: the un-fused calls copy them byte by byte, the low-latency calls refuse them."""
    T, H, E, K = 20, 256, 8, 2
    idx, w = _routing(T, E, K, seed=16)
    goes = (idx >= 0).any(1)
    buf = tm.Buffer(None, 0, low_latency_mode=True, explicitly_destroy=True)

    def shifted(*shape):
        n = torch.Size(shape).numel()
        return torch.randn(n + 1, device="cuda").to(torch.bfloat16)[1:].view(shape)
    x, y, out = shifted(T, H), shifted(E, T, H), shifted(T, H)
    recv, *_, handle, _ = buf.deepep_dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E)
    assert torch.equal(recv, x[goes]) and torch.equal(buf.deepep_combine(x[: recv.shape[0]], handle)[0][goes], x[: recv.shape[0]])
    with pytest.raises(RuntimeError, match="16-byte"):
        buf.low_latency_dispatch(x, idx, T, E, use_fp8=False)
    low = buf.low_latency_dispatch(x.clone(), idx, T, E, use_fp8=False)[2]
    with pytest.raises(RuntimeError, match="16-byte"):
        buf.low_latency_combine(y, idx, w, low)
    with pytest.raises(RuntimeError, match="16-byte"):
        buf.low_latency_combine(y.clone(), idx, w, low, out=out)
    buf.destroy()
