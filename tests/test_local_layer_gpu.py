"""The one-rank layer (csrc/local_layer.cu) against the kernels that several ranks use, bit for bit (same slots, tiles and order
of every sum), and against the fp32 oracle."""
import pytest
import torch

import teramoe_b200 as tm
from teramoe_b200.utils.numerics import assert_close_bf16
from helpers import make_problem, oracle

pytestmark = pytest.mark.gpu


def _run(buf, prob, idx, E, **kw):
    r = prob["ranks"][0]
    x = r["x"].clone().requires_grad_(True)
    w = r["w"].clone().requires_grad_(True)
    Wg = prob["W_gateup"].clone().requires_grad_(True)
    Wd = prob["W_down"].clone().requires_grad_(True)
    out = buf.teramoe_autograd(x, idx, w, Wg, Wd, E, **kw)
    out.backward(r["go"])
    fwd = buf.teramoe_forward(r["x"], idx, r["w"], prob["W_gateup"], prob["W_down"], E, **kw)
    torch.cuda.synchronize()
    return {"out": out.detach(), "dx": x.grad, "dw": w.grad, "dWg": Wg.grad, "dWd": Wd.grad, "forward only": fwd}


@pytest.mark.parametrize("T,H,I,E,K,skew,kw", [
    (1, 64, 64, 1, 1, False, {}),                        # the smallest sizes: one tile, mostly outside
    (3, 256, 128, 300, 8, False, {}),                    # far more experts than entries
    (128, 512, 192, 2, 2, False, {}),                    # exactly one full block per expert, half a column block
    (129, 320, 320, 2, 2, False, {}),                    # one row more
    (257, 1088, 704, 5, 3, True, {"stage": 2}),          # three chunks' worth of ragged segments, columns past every tile edge
    (512, 128, 64, 20, 8, False, {}),                    # the most entries that every routing block counts itself
    (513, 128, 64, 20, 8, False, {}),                    # one token more: chunk histograms
    (1000, 768, 640, 40, 32, False, {"compute_batch_size": 1024, "combine_start_head_percent": 0}),
    (2100, 512, 256, 8, 4, True, {"compute_batch_size": 4096, "combine_start_head_percent": 100, "total_sms": 64, "num_dispatch_sms": 8}),
])
def test_one_rank_layer_matches_general_kernels_and_oracle(T, H, I, E, K, skew, kw, monkeypatch):
    from teramoe_b200 import engine
    prob = make_problem(1, T, H, I, E, K, seed=T, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02, drop_some=T > 3)
    idx = prob["ranks"][0]["idx"]
    if skew:                                             # most tokens take expert 0 first; some go nowhere
        idx = idx.clone()
        idx[::2, 0] = 0
        idx[5::7] = -1
        dup = (idx[:, 1:] == 0) & (idx[:, :1] == 0)
        idx[:, 1:][dup] = -1
        prob["ranks"][0]["idx"] = idx
    if T == 1000:
        idx = idx.to(torch.int32)
    buf = tm.Buffer(None, int(64e6), explicitly_destroy=True)
    res = {}
    for mode in ("0", "auto"):
        monkeypatch.setattr(engine, "_LOCAL_LAYER_MODE", mode)
        for name in ("_FUSED_DISPATCH_MODE", "_FUSED_MODE", "_LAYER_KERNEL_MODE"):
            monkeypatch.setattr(engine, name, "1" if mode == "0" else "auto")
        res[mode] = [_run(buf, prob, idx, E, **kw) for _ in range(2)]
    ref = oracle(prob)[0]
    for name in ("out", "dx", "dw", "dWg", "dWd"):
        assert_close_bf16(res["auto"][0][name].float(), ref[name].cuda().float(), name)
    for name, got in res["auto"][0].items():
        assert torch.equal(got, res["auto"][1][name]), f"{name}: two runs differ"
        assert torch.equal(got, res["0"][0][name]), f"{name}: differs from the general kernels"
    buf.check_status()
    buf.destroy()


@pytest.mark.parametrize("H,I,copies", [
    (192, 128, (False, False)),                          # loading warps, two slices of columns and a half, and many
    (4160, 64, (False, False)),
    (192, 256, (False, True)),                           # rows copied several at once, and one after the other
    (4160, 256, (False, True)),
    (192, 4096, (True, True)),
    (4160, 4096, (True, True)),
])
def test_rows_per_expert_at_the_edges_of_operand_boxes(H, I, copies, monkeypatch):
    """An expert's rows are copied 8 at a time, loaded 32 at a time up to 64 and 128 at a time above (by loading warps 32 or 128), summed 16
    at a time, and stored 32 at a time."""
    from teramoe_b200 import engine
    from teramoe_b200._build import load_ext
    counts = [1, 0, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 161, 255, 256, 257]
    E, T = len(counts), sum(counts)
    train, forward = (load_ext().local_layer_variant(T, 1, E, H, I, keep) for keep in (True, False))
    assert (train["copies_forward"], train["copies_backward"], forward["copies_forward"], forward["few"]) == (*copies, copies[0], 0)
    prob = make_problem(1, T, H, I, E, 1, seed=3, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    order = torch.randperm(T, generator=torch.Generator().manual_seed(1))
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[order].view(T, 1).to(prob["ranks"][0]["idx"])
    prob["ranks"][0]["idx"] = idx
    buf = tm.Buffer(None, int(64e6), explicitly_destroy=True)
    res = {}
    for mode in ("0", "auto"):
        monkeypatch.setattr(engine, "_LOCAL_LAYER_MODE", mode)
        for name in ("_FUSED_DISPATCH_MODE", "_FUSED_MODE", "_LAYER_KERNEL_MODE"):
            monkeypatch.setattr(engine, name, "1" if mode == "0" else "auto")
        res[mode] = _run(buf, prob, idx, E)
    ref = oracle(prob)[0]
    for name, got in res["auto"].items():
        if name in ref:
            assert_close_bf16(got.float(), ref[name].cuda().float(), name)
        assert torch.equal(got, res["0"][name]), f"{name}: differs from the general kernels"
    buf.check_status()
    buf.destroy()


@pytest.mark.parametrize("counts,H,I,halves", [
    ([257, 300, 320, 321, 383, 384, 385, 641, 0], 192, 128, 1),      # half units behind whole ones: 1, 44, 64, 65, 127 and 128 rows of the last block
    ([257, 300, 320, 321, 383, 384, 385, 641, 0], 192, 1024, 1),     # (rows by copies in backward)
    ([257, 300, 320, 321, 383, 384, 385, 641, 0], 2112, 128, 0),     # the same with zeros for a second block
    ([257, 300, 320, 321, 383, 384, 385, 641, 0], 2112, 1024, 0),
    ([1, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128, 500], 2112, 4096, 1),
])
def test_last_units_of_experts(counts, H, I, halves, monkeypatch):
    from teramoe_b200 import engine
    from teramoe_b200._build import load_ext
    E, T = len(counts), sum(counts)
    assert load_ext().local_layer_halves(T, 1, E, H, I) == halves
    prob = make_problem(1, T, H, I, E, 1, seed=3, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    order = torch.randperm(T, generator=torch.Generator().manual_seed(1))
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[order].view(T, 1).to(prob["ranks"][0]["idx"])
    buf = tm.Buffer(None, int(64e6), explicitly_destroy=True)
    res = {}
    for mode in ("0", "auto"):
        monkeypatch.setattr(engine, "_LOCAL_LAYER_MODE", mode)
        for name in ("_FUSED_DISPATCH_MODE", "_FUSED_MODE", "_LAYER_KERNEL_MODE"):
            monkeypatch.setattr(engine, name, "1" if mode == "0" else "auto")
        res[mode] = [_run(buf, prob, idx, E) for _ in range(2)]
    for runs in zip(*res.values()):
        for name, got in runs[1].items():
            assert torch.equal(got, runs[0][name]), f"{name}: differs from the general kernels"
    buf.check_status()
    buf.destroy()


def test_last_units_of_experts_with_wide_tiles(monkeypatch):
    """Half units where every GEMM takes 512-column tiles (1344 = 2 * 512 + 320: a last one and a quarter): 1, 64, 65 and 128 rows in the last block."""
    from teramoe_b200 import engine
    from teramoe_b200._build import load_ext
    H, I, counts = 2048, 1344, [3840 + r for r in (1, 64, 65, 128, 0, 63, 96, 127, 1, 32, 33, 128)] + [2, 7700]
    E, T = len(counts), sum(counts)
    assert load_ext().local_layer_halves(T, 1, E, H, I) and load_ext().local_layer_columns(T, 1, E, H, I) == [[512] * 2, [512] * 4]
    prob = make_problem(1, T, H, I, E, 1, seed=3, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    order = torch.randperm(T, generator=torch.Generator().manual_seed(1))
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[order].view(T, 1).to(prob["ranks"][0]["idx"])
    buf = tm.Buffer(None, int(64e6), explicitly_destroy=True)
    res = {}
    for mode in ("0", "auto"):
        monkeypatch.setattr(engine, "_LOCAL_LAYER_MODE", mode)
        for name in ("_FUSED_DISPATCH_MODE", "_FUSED_MODE", "_LAYER_KERNEL_MODE"):
            monkeypatch.setattr(engine, name, "1" if mode == "0" else "auto")
        res[mode] = _run(buf, prob, idx, E)
    for name, got in res["auto"].items():
        assert torch.equal(got, res["0"][name]), f"{name}: differs from the general kernels"
    buf.check_status()
    buf.destroy()


@pytest.mark.parametrize("batch", [1024, 2048, 4096])
def test_batches_end_where_experts_do(batch, monkeypatch):
    """Experts of 9, 4, 1, 0, 2, 8, 3, 5 and 1 units of 256 rows in nominal batches of 4, 8 and 16: ends that move to an expert's, that stay inside
    one, and a tie."""
    from teramoe_b200 import engine
    counts = [9 * 256 - 100, 1024, 1, 0, 500, 2048, 513, 1200, 200]
    E, T = len(counts), sum(counts)
    prob = make_problem(1, T, 128, 64, E, 1, seed=5, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    order = torch.randperm(T, generator=torch.Generator().manual_seed(2))
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[order].view(T, 1).to(prob["ranks"][0]["idx"])
    buf = tm.Buffer(None, int(64e6), explicitly_destroy=True)
    res = {}
    for mode in ("0", "auto"):
        monkeypatch.setattr(engine, "_LOCAL_LAYER_MODE", mode)
        for name in ("_FUSED_DISPATCH_MODE", "_FUSED_MODE", "_LAYER_KERNEL_MODE"):
            monkeypatch.setattr(engine, name, "1" if mode == "0" else "auto")
        res[mode] = _run(buf, prob, idx, E, compute_batch_size=batch)
    for name, got in res["auto"].items():
        assert torch.equal(got, res["0"][name]), f"{name}: differs from the general kernels"
    buf.check_status()
    buf.destroy()


@pytest.mark.parametrize("H,I", [(512, 64), (64, 512), (1024, 128)])
def test_loading_warps_keep_up_with_short_items(H, I):
    """Items of one to a few steps of K, in which the loading warps have rows to bring and in which they have none, many times over: no
    step is left behind (its wait would run out) and every run gives the same bits."""
    prob = make_problem(1, 3000, H, I, 24, 4, seed=H, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    buf = tm.Buffer(None, int(64e6), explicitly_destroy=True)
    want = _run(buf, prob, prob["ranks"][0]["idx"], 24)
    for _ in range(30):
        got = _run(buf, prob, prob["ranks"][0]["idx"], 24)
        assert all(torch.equal(got[name], want[name]) for name in want)
    buf.check_status()
    buf.destroy()


@pytest.mark.parametrize("H,I", [(128, 64), (1024, 128)])         # one step of K after the other, and two turns through the stages
def test_rows_of_both_ctas_are_those_of_this_call(H, I, monkeypatch):
    """Units of 256 rows, half of them loaded by the second CTA, with other values in every call: an operand that is multiplied before it is
    there holds rows of another step or another call."""
    from teramoe_b200 import engine
    prob = make_problem(1, 2048, H, I, 8, 1, seed=H, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    r["idx"] = (torch.arange(2048, device="cuda") % 8).view(2048, 1)
    buf = tm.Buffer(None, int(64e6), explicitly_destroy=True)
    gen = torch.Generator(device="cuda").manual_seed(7)
    for _ in range(10):
        r["x"].normal_(0, 0.1, generator=gen)
        r["go"].normal_(0, 1.0, generator=gen)
        res = {}
        for mode in ("0", "auto"):
            monkeypatch.setattr(engine, "_LOCAL_LAYER_MODE", mode)
            for name in ("_FUSED_DISPATCH_MODE", "_FUSED_MODE", "_LAYER_KERNEL_MODE"):
                monkeypatch.setattr(engine, name, "1" if mode == "0" else "auto")
            res[mode] = _run(buf, prob, r["idx"], 8)
        for name, got in res["auto"].items():
            assert torch.equal(got, res["0"][name]), f"{name}: differs from the general kernels"
    buf.check_status()
    buf.destroy()


@pytest.mark.parametrize("counts,empty,H,I,K", [
    # rows around the multiples of 4 (row copies), 16 (columns of the accumulator) and 64 (units); a last tile of weights that is half outside
    ([1, 3, 4, 5, 15, 16, 17, 31, 33, 47, 63, 64, 65, 127, 128, 129, 2], 100, 192, 64, 2),
    ([1, 3, 4, 5, 15, 16, 17, 31, 33, 47, 63, 64, 65, 127, 128, 129, 2], 100, 1088, 320, 2),
    ([300], 60, 1088, 320, 2),                           # all rows on one expert, far more than the average
    ([64, 64, 1], 40, 512, 4096, 3),                     # I so large that other forwards copy rows
    ([70, 20, 9], 100, 320, 128, 9),                     # sums of more than eight entries, one at the end
    ([40, 33, 2], 200, 320, 128, 32),
])
def test_forward_with_few_rows_per_expert(counts, empty, H, I, K, monkeypatch):
    """Also: tokens without an expert; more blocks than tiles and the other way round."""
    from teramoe_b200 import engine
    from teramoe_b200._build import load_ext
    E, T = len(counts) + empty, sum(counts) + 3
    assert load_ext().local_layer_variant(T, K, E, H, I, False)["few"]
    gen = torch.Generator().manual_seed(1)
    experts = torch.repeat_interleave(torch.arange(len(counts)), torch.tensor(counts))
    idx = torch.full((T, K), -1, dtype=torch.int64)
    idx[torch.randperm(T, generator=gen)[: len(experts)], K - 1] = experts[torch.randperm(len(experts), generator=gen)]
    if K > 8:                                            # and for some tokens all entries
        idx[:2] = torch.randperm(E - len(counts), generator=gen)[:K] + len(counts)
    prob = make_problem(1, T, H, I, E, K, seed=8, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    idx = idx.cuda()
    buf = tm.Buffer(None, int(64e6), explicitly_destroy=True)
    res = {}
    for mode in ("0", "auto"):
        monkeypatch.setattr(engine, "_LOCAL_LAYER_MODE", mode)
        for name in ("_FUSED_DISPATCH_MODE", "_FUSED_MODE", "_LAYER_KERNEL_MODE"):
            monkeypatch.setattr(engine, name, "1" if mode == "0" else "auto")
        call = lambda i, **kw: buf.teramoe_forward(r["x"], i, r["w"], prob["W_gateup"], prob["W_down"], E, **kw)
        res[mode] = [call(idx), call(idx, total_sms=16, num_dispatch_sms=4, num_combine_sms=4), call(torch.full_like(idx, -1))]
    for got, want in zip(res["auto"], res["0"]):
        assert torch.equal(got, want)
    assert bool(res["auto"][0].any()) and not bool(res["auto"][2].any())
    buf.check_status()
    buf.destroy()


@pytest.mark.parametrize("T,K,E,total_sms", [(700, 2, 100, 6), (4096, 1, 256, 8)])
def test_few_rows_kernel_routes_on_a_grid_smaller_than_the_routing(T, K, E, total_sms, monkeypatch):
    """Eleven and twenty-four shares of the routing on six and eight blocks: each takes several, one after the other; tokens without an expert."""
    from teramoe_b200 import engine
    from teramoe_b200._build import load_ext
    H, I = 192, 128
    assert load_ext().local_layer_variant(T, K, E, H, I, False)["few"] == 1
    prob = make_problem(1, T, H, I, E, K, seed=T, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    idx = r["idx"].clone()
    idx[5::7] = -1
    buf = tm.Buffer(None, int(64e6), explicitly_destroy=True)
    call = lambda **kw: buf.teramoe_forward(r["x"], idx, r["w"], prob["W_gateup"], prob["W_down"], E, **kw)
    with monkeypatch.context() as m:
        m.setattr(engine, "_LOCAL_LAYER_MODE", "0")
        for name in ("_FUSED_DISPATCH_MODE", "_FUSED_MODE", "_LAYER_KERNEL_MODE"):
            m.setattr(engine, name, "1")
        want = call()
    for kw in (dict(total_sms=total_sms, num_dispatch_sms=2, num_combine_sms=2), {}):
        assert torch.equal(call(**kw), want) and buf._engine.native.ran_few()
    buf.check_status()
    buf.destroy()


@pytest.mark.parametrize("counts,E,T,H,I,few,ran", [
    ([70, 33, 15, 5], 8, 128, 320, 64, 1, True),         # units of 64 rows
    ([65, 64, 63, 33, 31, 17, 16, 15], 25, 307, 192, 256, 2, True),
    ([200, 50, 50], 25, 307, 1088, 320, 2, False),       # three units beyond the first ones of three experts
    ([100, 20, 5], 4, 128, 320, 64, 1, True),            # units of 128 rows
    ([60, 1], 3, 64, 320, 64, 1, True),                  # (not where there are no more tokens than 64)
    ([1, 15, 17, 33, 64, 65, 95, 96, 97, 127, 128, 129], 30, 870, 192, 1920, 2, True),      # a last tile of weights that is half outside
    ([1, 15, 17, 33, 64, 65, 95, 96, 97, 127, 128, 129], 30, 870, 1088, 1920, 2, True),
    ([257, 129, 128], 24, 520, 1088, 1408, 2, False),     # as many units beyond the first as experts
])
def test_forward_with_up_to_eighty_rows_per_expert(counts, E, T, H, I, few, ran, monkeypatch):
    """Rows at the edges of row copies (4), accumulator columns (16), reads of the accumulator (32) and units (64, 128); which kernel takes the
    call; twice, and on fewer SMs: the bits of the several-rank kernels each time."""
    from teramoe_b200 import engine
    from teramoe_b200._build import load_ext
    assert 16 * E < 2 * T <= 80 * E and load_ext().local_layer_variant(T, 2, E, H, I, False)["few"] == few
    idx = torch.full((T, 2), -1, dtype=torch.int64)
    idx[: sum(counts), 1] = torch.repeat_interleave(torch.arange(len(counts)), torch.tensor(counts))
    idx = idx[torch.randperm(T, generator=torch.Generator().manual_seed(1))].cuda()
    prob = make_problem(1, T, H, I, E, 2, seed=8, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    buf = tm.Buffer(None, int(64e6), explicitly_destroy=True)
    call = lambda **kw: buf.teramoe_forward(r["x"], idx, r["w"], prob["W_gateup"], prob["W_down"], E, **kw)
    with monkeypatch.context() as m:
        m.setattr(engine, "_LOCAL_LAYER_MODE", "0")
        for name in ("_FUSED_DISPATCH_MODE", "_FUSED_MODE", "_LAYER_KERNEL_MODE"):
            m.setattr(engine, name, "1")
        want = call()
    for kw in ({}, {}, dict(total_sms=16, num_dispatch_sms=4, num_combine_sms=4)):
        assert torch.equal(call(**kw), want) and buf._engine.native.ran_few() == ran
    buf.check_status()
    buf.destroy()


@pytest.mark.parametrize("counts,H,I,unit", [
    ([128, 128, 127, 97, 96, 95, 66, 65], 4096, 1024, 128),      # one turn of 128-row tiles, two of 64-row tiles
    ([128, 128, 127, 97, 96, 95, 66, 65], 4096, 512, 64),        # one turn of either
    ([128, 128, 128, 128, 0, 0, 0, 0], 7168, 512, 64),           # neither fills one
    ([128, 65, 64, 64, 33, 1, 0, 16], 4096, 1024, 64),           # few tiles more, and a large unit's steps
    ([70, 70, 70, 70, 70, 70, 70, 70], 1024, 1024, 64),          # small weights
])
def test_units_of_up_to_128_tokens_follow_the_routing(counts, H, I, unit, monkeypatch):
    """The kernel that routes by itself chooses the rows of a unit from the entries per expert, also when a captured call is replayed with other ones."""
    from teramoe_b200 import engine
    from teramoe_b200._build import load_ext
    T, K, E = 128, 8, 16
    assert load_ext().local_layer_variant(T, K, E, H, I, False)["few"] == 1
    gen = torch.Generator().manual_seed(2)
    idx = torch.full((T, K), -1, dtype=torch.int64)
    for e, n in enumerate(counts):
        idx[torch.randperm(T, generator=gen)[:n], e] = 2 * e
    prob = make_problem(1, T, H, I, E, K, seed=8, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    idx, even = idx.cuda(), (torch.arange(T * K, device="cuda") % E).view(T, K)      # even: 64 rows per expert
    buf = tm.Buffer(None, int(64e6), explicitly_destroy=True)
    call = lambda i: buf.teramoe_forward(r["x"], i, r["w"], prob["W_gateup"], prob["W_down"], E)
    with monkeypatch.context() as m:
        m.setattr(engine, "_LOCAL_LAYER_MODE", "0")
        for name in ("_FUSED_DISPATCH_MODE", "_FUSED_MODE", "_LAYER_KERNEL_MODE"):
            m.setattr(engine, name, "1")
        want, want_even = call(idx), call(even)
    for _ in range(2):
        assert torch.equal(call(idx), want)
        assert buf._engine.native.ran_few() and buf._engine.native.few_unit() == unit
    static = even.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call(static)
    for i, ref, rows in ((idx, want, unit), (even, want_even, 64), (idx, want, unit)):
        static.copy_(i)
        graph.replay()
        assert torch.equal(out, ref) and buf._engine.native.few_unit() == rows
    buf.check_status()
    buf.destroy()


@pytest.mark.parametrize("counts,H,I,few", [
    ([64] * 20 + [8] * 10, 4096, 1024, True),            # no second unit
    ([129] * 6 + [64] * 6, 4096, 1024, True),            # as many as experts with rows
    ([129] * 7 + [64] * 5 + [8], 4096, 1024, False),     # one more
    ([700], 4096, 1024, False),                          # all rows on one expert
    ([700], 512, 256, True),                             # so small a layer that it does not matter
])
def test_forward_with_few_rows_on_average_by_their_spread(counts, H, I, few, monkeypatch):
    """Which kernel takes a call is decided by the routing, on the GPU: also when a captured call is replayed with other indices."""
    from teramoe_b200 import engine
    from teramoe_b200._build import load_ext
    T = sum(counts) + 3
    E = max(-(-2 * T // 16), len(counts))
    assert load_ext().local_layer_variant(T, 2, E, H, I, False)["few"] == (2 if H > 512 else 1)
    idx = torch.full((T, 2), -1, dtype=torch.int64)
    idx[: sum(counts), 0] = torch.repeat_interleave(torch.arange(len(counts)), torch.tensor(counts))
    idx = idx[torch.randperm(T, generator=torch.Generator().manual_seed(1))].cuda()
    even = (torch.arange(2 * T, device="cuda") % E).view(T, 2)
    prob = make_problem(1, T, H, I, E, 2, seed=8, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    buf = tm.Buffer(None, int(64e6), explicitly_destroy=True)
    call = lambda i: buf.teramoe_forward(r["x"], i, r["w"], prob["W_gateup"], prob["W_down"], E)
    with monkeypatch.context() as m:
        m.setattr(engine, "_LOCAL_LAYER_MODE", "0")
        for name in ("_FUSED_DISPATCH_MODE", "_FUSED_MODE", "_LAYER_KERNEL_MODE"):
            m.setattr(engine, name, "1")
        want, want_even = call(idx), call(even)
    ran_few = buf._engine.native.ran_few
    for i, ref, kernel in ((idx, want, few), (even, want_even, True)):
        assert torch.equal(call(i), ref) and ran_few() == kernel
    static = even.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call(static)
    for i, ref, kernel in ((idx, want, few), (even, want_even, True), (idx, want, few)):
        static.copy_(i)
        graph.replay()
        assert torch.equal(out, ref) and ran_few() == kernel
    buf.check_status()
    buf.destroy()


@pytest.mark.parametrize("T,H,I,E,K,copies", [
    (511, 192, 512, 4, 2, (False, True)),                # 255 rows per expert on average, below half of I: copies in backward
    (512, 192, 512, 4, 2, (False, False)),               # at half of it: loading warps
    (700, 320, 4032, 3, 2, (False, True)),
    (700, 320, 4096, 3, 2, (True, True)),                # I so large that rows are copied in both directions
])
def test_rows_by_copies_and_by_loading_warps(T, H, I, E, K, copies, monkeypatch):
    """Both sides of the rule that says how token rows become operands."""
    from teramoe_b200 import engine
    from teramoe_b200._build import load_ext
    variant = load_ext().local_layer_variant(T, K, E, H, I, True)
    assert (variant["copies_forward"], variant["copies_backward"]) == copies
    prob = make_problem(1, T, H, I, E, K, seed=T, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02, drop_some=False)
    buf = tm.Buffer(None, int(64e6), explicitly_destroy=True)
    res = {}
    for mode in ("0", "auto"):
        monkeypatch.setattr(engine, "_LOCAL_LAYER_MODE", mode)
        for name in ("_FUSED_DISPATCH_MODE", "_FUSED_MODE", "_LAYER_KERNEL_MODE"):
            monkeypatch.setattr(engine, name, "1" if mode == "0" else "auto")
        res[mode] = _run(buf, prob, prob["ranks"][0]["idx"], E)
    for name, got in res["auto"].items():
        assert torch.equal(got, res["0"][name]), f"{name}: differs from the general kernels"
    buf.check_status()
    buf.destroy()


def test_native_autograd_node_keeps_its_buffer_and_fills_the_given_gradient():
    """The buffer may go out of scope before the backward pass; d(topk_weights) goes to the caller's tensor; a second derivative
    raises; a destroyed buffer raises."""
    prob = make_problem(1, 200, 512, 256, 8, 2, seed=4, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    Wg, Wd = prob["W_gateup"].requires_grad_(True), prob["W_down"].requires_grad_(True)
    grads = []
    for given in (None, torch.full((200, 2), 7.0, device="cuda")):
        x, w = r["x"].clone().requires_grad_(True), r["w"].clone().requires_grad_(True)
        out = tm.Buffer(None, 0).teramoe_autograd(x, r["idx"], w, Wg, Wd, 8, grad_topk_weights=given)
        out.backward(r["go"])
        grads.append((x.grad, w.grad))
        if given is not None:
            assert torch.equal(given, w.grad)
    assert torch.equal(grads[0][0], grads[1][0]) and torch.equal(grads[0][1], grads[1][1])
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    x = r["x"].clone().requires_grad_(True)
    out = buf.teramoe_autograd(x, r["idx"], r["w"], Wg, Wd, 8)
    (dx,) = torch.autograd.grad(out, x, r["go"].clone().requires_grad_(True), create_graph=True)
    assert torch.equal(dx, grads[0][0])
    with pytest.raises(RuntimeError, match="once_differentiable"):
        dx.float().sum().backward()
    out = buf.teramoe_autograd(x, r["idx"], r["w"], Wg, Wd, 8)
    buf.destroy()
    with pytest.raises(RuntimeError, match="destroyed"):
        out.backward(r["go"])


def test_second_backward_of_one_forward_raises():
    """The workspace of a forward serves one backward pass: a second one raises, with and without retain_graph, on this path as on the
    several-rank kernels, and a call that was refused before it reached the GPU does not count."""
    prob = make_problem(1, 200, 512, 256, 8, 2, seed=4, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    leaves = [r["x"].clone().requires_grad_(True), r["w"].clone().requires_grad_(True), prob["W_gateup"].requires_grad_(True),
              prob["W_down"].requires_grad_(True)]

    def forward():
        return buf.teramoe_autograd(leaves[0], r["idx"], leaves[1], leaves[2], leaves[3], 8)
    want = torch.autograd.grad(forward(), leaves, r["go"])
    for keep in (False, True):
        out = forward()
        buf._world.status[0] = 1                        # a report of an earlier call is raised before anything is launched ...
        buf._world._status_host[0] = 1
        with pytest.raises(RuntimeError, match="ran out"):
            torch.autograd.grad(out, leaves, r["go"], retain_graph=True)
        got = torch.autograd.grad(out, leaves, r["go"], retain_graph=keep)        # ... so this is the first pass
        for a, b in zip(got, want):
            assert torch.equal(a, b)
        with pytest.raises(RuntimeError, match="second"):
            torch.autograd.grad(out, leaves, r["go"])
    buf.check_status()
    buf.destroy()


def test_activation_and_its_gradient_over_the_range_of_the_gate(monkeypatch):
    """One expert with W_down = identity and gate = x[0], up = x[1] for every column: `out` is the activation itself and dx its two
    derivatives (64 equal terms).  Against the formulas in 64 bits; silu(g) and its derivative, computed by CUDA's functions, are within
    their documented errors (a few ulp of 32 bits) far below bf16, whose rounding (2^-9 each of preact, act and result) bounds the rest."""
    from teramoe_b200 import engine
    g = torch.cat([s * torch.logspace(-38, 4, 300, dtype=torch.float64) for s in (1.0, -1.0)] + [torch.linspace(-100, 100, 401, dtype=torch.float64),
                  torch.zeros(1, dtype=torch.float64), torch.linspace(-89, -85, 33, dtype=torch.float64)])
    T, H, I = g.numel(), 64, 64
    u = torch.tensor([1.0, -0.75, 3.0], dtype=torch.float64).repeat(T)[:T]
    x = torch.zeros(T, H)
    x[:, 0], x[:, 1] = g, u
    x = x.to(torch.bfloat16).cuda()
    g, u = x[:, 0].double(), x[:, 1].double()
    Wg = torch.zeros(1, 2 * I, H, device="cuda", dtype=torch.bfloat16)
    Wg[0, 0::2, 0] = 1.0
    Wg[0, 1::2, 1] = 1.0
    Wd = torch.eye(I, device="cuda", dtype=torch.bfloat16).view(1, H, I).contiguous()
    idx, w = torch.zeros(T, 1, dtype=torch.int64, device="cuda"), torch.full((T, 1), 0.5, device="cuda")
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    res = []
    for mode in ("0", "auto"):
        monkeypatch.setattr(engine, "_LOCAL_LAYER_MODE", mode)
        leaf = x.clone().requires_grad_(True)
        out = buf.teramoe_autograd(leaf, idx, w, Wg, Wd, 1)
        out.backward(torch.ones_like(out))
        res.append((out.detach(), leaf.grad))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
    out, dx = res[1]
    sig = torch.sigmoid(g)
    s = g * sig
    tiny = 1e-35                                      # where 1 + e^-g leaves the range of the fast division, and below the normal numbers
    want = 0.5 * s * u
    assert bool(((out[:, 0].double() - want).abs() <= 2.0 ** -8 * want.abs() + tiny).all())
    assert torch.equal(out, out[:, :1].expand_as(out))
    d_gate, d_up = (sig - s * sig + s) * 0.5 * u, 0.5 * s
    size = (sig + (s * sig).abs() + s.abs()) * 0.5 * u.abs()      # terms of the derivative, which cancel around g = -1.28
    assert bool(((dx[:, 0].double() / I - d_gate).abs() <= 2.0 ** -8 * d_gate.abs() + 2.0 ** -20 * size + tiny).all())
    assert bool(((dx[:, 1].double() / I - d_up).abs() <= 2.0 ** -8 * d_up.abs() + tiny).all())
    buf.destroy()


def test_schedule_arguments_may_be_floats():
    prob = make_problem(1, 200, 512, 256, 8, 2, seed=4, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    call = lambda **kw: buf.teramoe_forward(r["x"], r["idx"], r["w"], prob["W_gateup"], prob["W_down"], 8, **kw)
    want = call()
    for kw in ({"combine_start_head_percent": 55.5}, {"compute_batch_size": 1024.0, "combine_start_head_percent": 41}, {"total_sms": 100.0}):
        assert torch.equal(call(**kw), want)
    assert buf._engine.last_paths.get("layer_kernel", False)
    buf.destroy()


def test_forward_mode_and_function_transforms_raise():
    """There is no forward-mode derivative and no batching rule: both raise, with and without tensors that require a gradient."""
    import torch.autograd.forward_ad as fwad
    prob = make_problem(1, 64, 256, 128, 4, 2, seed=4, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    tensors = [r["x"], r["w"], prob["W_gateup"], prob["W_down"]]
    call = lambda x, w, wg, wd: buf.teramoe_autograd(x, r["idx"], w, wg, wd, 4)
    for i in range(4):
        for leaf in (False, True):
            with fwad.dual_level(), pytest.raises(NotImplementedError):
                args = [t.clone().requires_grad_(leaf and j == i) for j, t in enumerate(tensors)]
                args[i] = fwad.make_dual(args[i], torch.ones_like(args[i]))
                call(*args)
    for transform in (lambda f: torch.func.grad(f)(tensors[0]), lambda f: torch.func.vmap(f)(tensors[0][None]),
                      lambda f: torch.func.jvp(f, (tensors[0],), (tensors[0],))):
        with pytest.raises(RuntimeError):
            transform(lambda x: call(x, *tensors[1:]).float().sum())
    assert torch.equal(call(*tensors), buf.teramoe_forward(tensors[0], r["idx"], *tensors[1:], 4))
    buf.check_status()
    buf.destroy()


def test_launches_of_a_call():
    """Routing is one kernel up to 4096 entries and two above, each direction of the layer one."""
    from teramoe_b200._build import load_ext
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    for T, forward in ((2048, 2), (2049, 3)):
        prob = make_problem(1, T, 128, 64, 4, 2, seed=4, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
        r = prob["ranks"][0]
        x = r["x"].clone().requires_grad_(True)
        n = [load_ext().launch_count()]
        out = buf.teramoe_autograd(x, r["idx"], r["w"], prob["W_gateup"], prob["W_down"], 4)
        n.append(load_ext().launch_count())
        out.backward(r["go"])
        n.append(load_ext().launch_count())
        assert [b - a for a, b in zip(n, n[1:])] == [forward, 1]
    buf.check_status()
    buf.destroy()


def test_hooks_on_saved_tensors_see_no_workspace():
    """Hooks get the weights and the kept rows, which they may store elsewhere, recompute (activation checkpointing) or round; a hook that
    cannot take integers still works, and one that returns something else than it was given raises."""
    from torch.utils.checkpoint import checkpoint
    prob = make_problem(1, 200, 512, 256, 8, 2, seed=4, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    leaves = [r["x"].clone().requires_grad_(True), r["w"].clone().requires_grad_(True), prob["W_gateup"].requires_grad_(True),
              prob["W_down"].requires_grad_(True)]

    def forward(*a):
        return buf.teramoe_autograd(a[0], r["idx"], a[1], a[2], a[3], 8)
    want = torch.autograd.grad(forward(*leaves), leaves, r["go"])
    seen = []

    def pack(t):
        seen.append(t.dtype)
        return (t.float() * 2).cpu()
    hooks = torch.autograd.graph.saved_tensors_hooks
    with hooks(pack, lambda t: (t / 2).to(torch.bfloat16).cuda()):
        out = forward(*leaves)
    got = [torch.autograd.grad(out, leaves, r["go"])]
    assert seen == [torch.bfloat16] * 3
    got.append(torch.autograd.grad(checkpoint(forward, *leaves, use_reentrant=False), leaves, r["go"]))
    with torch.autograd.graph.save_on_cpu(pin_memory=True):
        out = forward(*leaves)
    got.append(torch.autograd.grad(out, leaves, r["go"]))
    for g in got:
        assert all(torch.equal(a, b) for a, b in zip(g, want))
    for wrong in (lambda t: t.float(), lambda t: t.cpu(), lambda t: t[..., :-1]):
        with hooks(lambda t: t, wrong):
            out = forward(*leaves)
        with pytest.raises(RuntimeError):
            torch.autograd.grad(out, leaves, r["go"])
    # only the rows are returned in another form
    rows = lambda t: t.dim() == 1
    for wrong in (lambda t: t.float(), lambda t: t.cpu(), lambda t: t[:-1], lambda t: t.repeat_interleave(2)[::2],
                  lambda t: torch.cat([t[:1], t])[1:]):
        with hooks(lambda t: t, lambda t, wrong=wrong: wrong(t) if rows(t) else t):
            out = forward(*leaves)
        with pytest.raises(RuntimeError, match="saved tensors"):
            torch.autograd.grad(out, leaves, r["go"])
    buf.check_status()
    buf.destroy()


@pytest.mark.parametrize("T,E,few", [(1, 16, True), (32, 16, True), (512, 16, False)])
def test_a_forward_reports_its_spans_and_waits(T, E, few):
    """Every forward replaces the report of the one before, and its time stamps lie in the order of the work."""
    from teramoe_b200._build import load_ext
    assert bool(load_ext().local_layer_variant(T, 8, E, 4096, 1024, False)["few"]) == few
    prob = make_problem(1, T, 4096, 1024, E, 8, seed=7, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    call = lambda i: buf.teramoe_forward(r["x"], i, r["w"], prob["W_gateup"], prob["W_down"], E)
    call(r["idx"])
    rep = buf._engine.wait_report()["fwd"]
    spans = rep["spans_ms"]
    assert set(spans) == {"gemm1", "gemm2", "reduce"}
    assert all(0 <= a <= b < 100 for a, b in spans.values())
    # (the clock ticks once in a microsecond or so)
    assert spans["gemm1"][0] == 0 <= spans["gemm2"][0] < spans["reduce"][0] and 0 < spans["gemm1"][1] < spans["gemm2"][1] <= spans["reduce"][1]
    assert rep["wait_arrival"] == rep["wait_wgrad"] == 0 and min(rep["wait_first_gemm"], rep["wait_landed"]) >= 0
    assert T == 1 or (rep["wait_first_gemm"] > 0 and rep["wait_landed"] > 0)
    call(torch.full_like(r["idx"], -1))
    assert set(buf._engine.wait_report()["fwd"]["spans_ms"]) == {"reduce"}
    buf.destroy()


def test_waits_of_a_forward_with_few_rows_that_run_out_are_reported():
    """With a limit of a nanosecond every wait for another block's tiles runs out: the kernel ends in order, the report is raised, and the buffer
    can be used again."""
    prob = make_problem(1, 32, 4096, 1024, 16, 8, seed=7, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    call = lambda: buf.teramoe_forward(r["x"], r["idx"], r["w"], prob["W_gateup"], prob["W_down"], 16)
    want = call()
    limit = buf._world.status[4:6]
    limit[0] = 1
    call()
    with pytest.raises(RuntimeError, match="flag wait"):
        buf.check_status()
    limit[0] = 0
    assert torch.equal(call(), want)
    buf.check_status()
    buf.destroy()


@pytest.mark.parametrize("I,copies", [(256, True), (128, False)])
def test_a_wait_that_runs_out_is_reported_and_the_next_call_works(I, copies):
    """A slot table that says less than the work list lets a block's rows never arrive: the wait for their copies runs out behind the early
    loads of weights, or the loading warps see it at once; the kernel ends in order, the report is raised, and the buffer can be used again."""
    from teramoe_b200._build import load_ext
    T, H, E = 128, 512, 2
    assert load_ext().local_layer_variant(T, 1, E, H, I, True)["copies_backward"] == copies
    prob = make_problem(1, T, H, I, E, 1, seed=7, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    idx = (torch.arange(T, device="cuda") // 64).view(T, 1)
    leaves = [r["x"].clone().requires_grad_(True), prob["W_gateup"].requires_grad_(True), prob["W_down"].requires_grad_(True)]
    buf = tm.Buffer(None, 0, explicitly_destroy=True)

    def forward():
        return buf.teramoe_autograd(leaves[0], idx, r["w"], leaves[1], leaves[2], E)
    want = torch.autograd.grad(forward(), leaves, r["go"])
    out = forward()
    torch.cuda.synchronize()
    ws = torch.empty(0, dtype=torch.int32, device="cuda").set_(buf._engine.native.stats(0).untyped_storage())      # tables of that forward
    slots = list(range(64)) + [-1] * 64 + list(range(64, 128)) + [-1] * 64
    words = ws.tolist()
    at = [i for i in range(len(words) - 256) if words[i] == 0 and words[i:i + 256] == slots]
    assert len(at) == 1
    ws[at[0]] = -1                                    # the first 64 rows are not copied (or the first is not there)
    buf.set_wait_limit_ms(20)
    torch.autograd.grad(out, leaves, r["go"])
    with pytest.raises(RuntimeError, match="flag wait"):
        buf.check_status()
    buf.set_wait_limit_ms(0)
    got = torch.autograd.grad(forward(), leaves, r["go"])
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    buf.check_status()
    buf.destroy()


def test_backward_next_to_a_growing_arena():
    """One thread runs backward passes, which need no interpreter lock, while this one replaces the arena under them."""
    import threading
    prob = make_problem(1, 300, 512, 256, 8, 2, seed=6, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02)
    r = prob["ranks"][0]
    buf = tm.Buffer(None, 0, explicitly_destroy=True)
    leaves = [r["x"].clone().requires_grad_(True), prob["W_gateup"].requires_grad_(True), prob["W_down"].requires_grad_(True)]
    outs = [buf.teramoe_autograd(leaves[0], r["idx"], r["w"], leaves[1], leaves[2], 8) for _ in range(40)]
    torch.cuda.synchronize()
    got = []
    thread = threading.Thread(target=lambda: got.extend(torch.autograd.grad(o, leaves, r["go"]) for o in outs))
    thread.start()
    for _ in range(6):
        buf._world.ensure_data(buf._world.data_bytes + (1 << 20))
    thread.join()
    torch.cuda.synchronize()
    assert len(got) == len(outs)
    for g in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(g, got[0]))
    buf.check_status()
    buf.destroy()


def test_wide_tiles_match_general_kernels(monkeypatch):
    """Sizes at which every GEMM takes 512-column tiles, with a last tile of one half (4160 = 8 * 512 + 64) and of one and a quarter
    (1344 = 2 * 512 + 320)."""
    from teramoe_b200 import engine
    prob = make_problem(1, 6000, 4160, 1344, 8, 4, seed=9, dtype=torch.bfloat16, device="cuda", x_scale=0.1, w_scale=0.02, drop_some=True)
    buf = tm.Buffer(None, int(64e6), explicitly_destroy=True)
    res = {}
    for mode in ("0", "auto"):
        monkeypatch.setattr(engine, "_LOCAL_LAYER_MODE", mode)
        for name in ("_FUSED_DISPATCH_MODE", "_FUSED_MODE", "_LAYER_KERNEL_MODE"):
            monkeypatch.setattr(engine, name, "1" if mode == "0" else "auto")
        res[mode] = _run(buf, prob, prob["ranks"][0]["idx"], 8)
    for name, got in res["auto"].items():
        assert torch.equal(got, res["0"][name]), f"{name}: differs from the general kernels"
    buf.check_status()
    buf.destroy()
