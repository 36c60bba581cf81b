"""GPU: the kernels at the sizes where a tile, a chunk or a dispatch rule ends, against the CPU oracle."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from oracle import experts as OE
from oracle import quant as OQ
from oracle import routing as OR
from tests.util import assert_close_moe

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fg():
    import flaggems_sglang_b200 as fg

    return fg


@pytest.fixture(autouse=True)
def _device_status():
    yield
    from flaggems_sglang_b200 import _C

    _C.check_device_status()


def _layer(T, H, I, E, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16)
    w1 = (torch.randn(E, 2 * I, H, generator=g) * H ** -0.5).to(torch.bfloat16)
    w2 = (torch.randn(E, H, I, generator=g) * I ** -0.5).to(torch.bfloat16)
    return x, w1, w2, g


# rows per expert around the edges of 8-row groups and of the 64-, 128- and 256-token tiles; the mean picks the tile
ROWS = {"64": [1, 0, 7, 8, 9, 15, 16, 17, 31, 33, 63, 64, 65, 80], "128": [1, 63, 64, 65, 127, 128, 129, 0],
        "256": [1, 127, 129, 255, 256, 257, 400, 513],
        # e4m3 block scales: experts on both sides of the line between the narrow and the wide kernel
        "mixed": [63, 64, 65, 0, 1, 300, 66, 17, 128]}


@pytest.mark.parametrize("tile", ROWS)
@pytest.mark.parametrize("kind", ["bf16", "n_major", "bias", "channel", "block"])
def test_rows_per_expert_at_tile_edges(fg, tile, kind):
    """CTA-pair GEMMs: every expert's last token tile is cut by its row count.  I and H leave a part-filled weight tile."""
    rows = ROWS[tile]
    E, T = len(rows), sum(rows)
    H, I = (384, 384) if kind == "block" else (320, 352)
    x, w1, w2, g = _layer(T, H, I, E, 7)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(rows))[torch.randperm(T, generator=g)].to(torch.int32).view(T, 1)
    tw = torch.rand(T, 1, generator=g) + 0.5
    xd, twd, idd = x.cuda(), tw.cuda(), ids.cuda()
    if kind in ("bf16", "bias"):
        kw, okw = dict(variant="tcgen05"), {}
        ref = OE.fused_experts(x, w1, w2, tw, ids)
        if kind == "bias":
            b1, b2 = torch.randn(E, 2 * I, generator=g), torch.randn(E, H, generator=g)
            kw.update(b1=b1.cuda(), b2=b2.cuda(), activation="swiglu_oai", gemm1_clamp_limit=7.0)
            ref = OE.fused_experts_with_bias(x, w1, b1, w2, b2, tw, ids, limit=7.0)
        out = fg.fused_experts(xd, w1.cuda(), w2.cuda(), twd, idd, **kw)
    elif kind == "n_major":
        out = fg.fused_experts(xd, w1.transpose(1, 2).contiguous().cuda(), w2.transpose(1, 2).contiguous().cuda(), twd, idd,
                               weights_n_major=True)
        ref = OE.fused_experts(x, w1, w2, tw, ids)
    else:
        q = OQ.quant_weight_per_channel if kind == "channel" else OQ.quant_weight_block128
        (w1q, w1s), (w2q, w2s) = q(w1), q(w2)
        kw = dict(per_channel_quant=True) if kind == "channel" else dict(block_shape=[128, 128], variant="tcgen05")
        out = fg.fused_experts(xd, w1q.cuda(), w2q.cuda(), twd, idd, use_fp8_w8a8=True, w1_scale=w1s.cuda(),
                               w2_scale=w2s.cuda(), **kw)
        ref = (OE.fused_experts_fp8_per_channel if kind == "channel" else OE.fused_experts_fp8)(x, w1q, w1s, w2q, w2s, tw, ids)
    assert_close_moe(out, ref, "fp8" if kind in ("channel", "block") else "bf16", f"{kind} tile {tile}")


@pytest.mark.parametrize("H,I", [(128, 9600), (19200, 128)])
@pytest.mark.parametrize("kind", ["bf16", "block"])
def test_many_tiles_per_worker(fg, H, I, kind):
    """CTA-pair GEMMs (gate/up, then down) whose workers have 65 tiles each: their list of tiles is refilled twice."""
    E = 64
    x, w1, w2, g = _layer(E + 32, H, I, E, 9)
    ids = torch.cat([torch.arange(E), torch.arange(32)]).to(torch.int32).view(-1, 1)
    tw = torch.rand(E + 32, 1, generator=g) + 0.5
    if kind == "bf16":
        out = fg.fused_experts(x.cuda(), w1.cuda(), w2.cuda(), tw.cuda(), ids.cuda(), variant="tcgen05")
        ref = OE.fused_experts(x, w1, w2, tw, ids)
    else:
        (w1q, w1s), (w2q, w2s) = OQ.quant_weight_block128(w1), OQ.quant_weight_block128(w2)
        out = fg.fused_experts(x.cuda(), w1q.cuda(), w2q.cuda(), tw.cuda(), ids.cuda(), use_fp8_w8a8=True, w1_scale=w1s.cuda(),
                               w2_scale=w2s.cuda(), block_shape=[128, 128], variant="tcgen05")
        ref = OE.fused_experts_fp8(x, w1q, w1s, w2q, w2s, tw, ids)
    assert_close_moe(out, ref, "fp8" if kind == "block" else "bf16", f"{kind} H={H} I={I}")


@pytest.mark.parametrize("gated", [True, False])
def test_wide_e4m3_kernel_stores_to_rows_at_16_bytes(fg, gated):
    """The wide block-scale kernel stores 32 bytes at a time where the output is aligned to that, and 16 where it is not: the
    same bits."""
    from flaggems_sglang_b200 import _C
    from flaggems_sglang_b200.ops.fused_moe import _gemm_args

    g = torch.Generator().manual_seed(3)
    rows, n, k = [70, 0, 300, 129], 384, 256
    E, numel = len(rows), sum(rows)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(rows)).to(torch.int32).view(-1, 1).cuda()
    sorted_ids, expert_ids, num_post = fg.moe_align_block_size(ids, 128, E)
    cap = sorted_ids.numel()
    a = torch.randn(cap, k, generator=g).to(torch.float8_e4m3fn).cuda()
    w = torch.randn(E, (2 if gated else 1) * n, k, generator=g).to(torch.float8_e4m3fn).cuda()
    a_scale, w_scale = torch.rand(cap, k // 128, generator=g).cuda(), torch.rand(E, w.shape[1] // 128, k // 128, generator=g).cuda()
    out_rows, outs = cap if gated else numel, []
    for shift in (0, 8, 16):  # bf16 elements
        buf = torch.zeros(out_rows * n + 16, dtype=torch.bfloat16, device="cuda")
        args = _gemm_args(variant=_C.VARIANTS["tcgen05"], activation=0, num_experts=E, top_k=1, block_size=128, numel=numel,
                          sorted_cap=cap, max_blocks=cap // 128, sorted_token_ids=sorted_ids.data_ptr(),
                          expert_ids=expert_ids.data_ptr(), num_tokens_post_padded=num_post.data_ptr(), dtype=_C.E4M3,
                          out_dtype=_C.BF16, n=n, k=k, a_rows=cap, a=a.data_ptr(), a_scale=a_scale.data_ptr(), w=w.data_ptr(),
                          w_scale=w_scale.data_ptr(), out=buf[shift:].data_ptr())
        lib = _C.lib()
        _C.check((lib.fmoe_gemm1_silu if gated else lib.fmoe_gemm2)(args, _C.stream_ptr()))
        outs.append(buf[shift:shift + out_rows * n].clone())
    assert float(outs[0].float().abs().sum()) > 0
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


# then 73 tiles a worker in the gate/up GEMM or in the down GEMM: every ring and list wraps round, both kinds of tile in turn
@pytest.mark.parametrize("H,I,per_worker", [(128, 256, 1), (256, 128, 1), (128, 12800, 64), (25600, 128, 64), (384, 6528, 32)])
def test_wide_e4m3_kernel_mixes_tile_heights(fg, H, I, per_worker):
    """Block-scale layers whose experts end in tiles of M = 128 and of M = 256, one to three K blocks long: the warps that share a
    quantisation group change from tile to tile, and a tile is over before the slowest warp has left the one before."""
    rows = [300, 65, 129, 256, 400, 128, 257, 640, 70, 512, 0, 384] * 3
    E, T = len(rows), sum(rows)
    workers, tiles = fg._C.lib().fmoe_sm_count() // 2, sum(-(-r // 256) for r in rows) * max(I // 128, H // 256)
    if per_worker > 1:
        assert tiles > per_worker * workers
    x, w1, w2, g = _layer(T, H, I, E, 11)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(rows))[torch.randperm(T, generator=g)].to(torch.int32).view(T, 1)
    tw = torch.rand(T, 1, generator=g) + 0.5
    (w1q, w1s), (w2q, w2s) = OQ.quant_weight_block128(w1), OQ.quant_weight_block128(w2)
    d = [v.cuda() for v in (x, w1q, w2q, tw, ids, w1s, w2s)]
    outs = [fg.fused_experts(*d[:5], use_fp8_w8a8=True, w1_scale=d[5], w2_scale=d[6], block_shape=[128, 128]) for _ in range(3)]
    assert_close_moe(outs[0], OE.fused_experts_fp8(x, w1q, w1s, w2q, w2s, tw, ids), "fp8", f"H={H} I={I}")
    assert all(torch.equal(o, outs[0]) for o in outs)


def test_e4m3_kernels_without_the_register_move(tmp_path):
    """The e4m3 block-scale kernels as they are launched where the compiler left too few registers for setmaxnreg: same sums
    in the same order, so the same bits."""
    code = """
import sys, torch
import flaggems_sglang_b200 as fg
g = torch.Generator(device="cuda").manual_seed(1)
E, H, I, k, outs = 8, 512, 384, 2, []
w1, w2 = (torch.randn(E, *s, generator=g, device="cuda") * s[1] ** -0.5 for s in ((2 * I, H), (H, I)))
q = [fg.quant_weight_block128(torch.cat(list(w))) for w in (w1, w2)]
w1q, s1 = q[0][0].view(E, 2 * I, H), q[0][1].view(E, 2 * I // 128, H // 128)
w2q, s2 = q[1][0].view(E, H, I), q[1][1].view(E, H // 128, I // 128)
for T in (20, 300, 900):
    x, logits = torch.randn(T, H, generator=g, device="cuda").bfloat16(), torch.randn(T, E, generator=g, device="cuda")
    outs.append(fg.fused_moe(x, w1q, w2q, logits, k, True, use_fp8_w8a8=True, w1_scale=s1, w2_scale=s2,
                             block_shape=[128, 128], variant="tcgen05").cpu())
fg._C.check_device_status()
torch.save(outs, sys.argv[1])
"""
    outs = []
    for move in ("1", "0"):
        path = str(tmp_path / f"out{move}.pt")
        env = dict(os.environ, FMOE_FOLD_MOVE_REGISTERS=move, PYTHONPATH=os.pathsep.join(sys.path))
        subprocess.run([sys.executable, "-c", code, path], check=True, env=env, timeout=300)
        outs.append(torch.load(path))
    assert all(torch.equal(a, b) for a, b in zip(*outs))


@pytest.mark.parametrize("T", [1, 2, 3, 5, 8, 9])
@pytest.mark.parametrize("kind", ["bf16", "bias", "block"])
def test_decode_layer(fg, T, kind):
    """Up to 8 tokens run in the two decode kernels (T = 9 is the first call that does not): shared experts, ids outside
    the range, and the router inside the call."""
    E, H, I, k = 16, 640, 384, 4
    x, w1, w2, g = _layer(T, H, I, E, 20 + T)
    logits = torch.randn(T, E, generator=g)
    tw, ids = OR.softmax_topk(logits, k, True)
    kw, wts = {}, (w1, w2)
    if kind == "block":
        (w1q, w1s), (w2q, w2s) = OQ.quant_weight_block128(w1), OQ.quant_weight_block128(w2)
        wts, kw = (w1q, w2q), dict(use_fp8_w8a8=True, w1_scale=w1s.cuda(), w2_scale=w2s.cuda(), block_shape=[128, 128])
        oracle = lambda w, i, **o: OE.fused_experts_fp8(x, w1q, w1s, w2q, w2s, w, i, **o)  # noqa: E731
    elif kind == "bias":
        b1, b2 = torch.randn(E, 2 * I, generator=g), torch.randn(E, H, generator=g)
        kw = dict(b1=b1.cuda(), b2=b2.cuda(), activation="swiglu_oai", gemm1_clamp_limit=7.0)
        oracle = lambda w, i, **o: OE.fused_experts_with_bias(x, w1, b1, w2, b2, w, i, limit=7.0, **o)  # noqa: E731
    else:
        oracle = lambda w, i, **o: OE.fused_experts(x, w1, w2, w, i, **o)  # noqa: E731
    d = [x.cuda(), wts[0].cuda(), wts[1].cuda()]
    tol = "fp8" if kind == "block" else "bf16"
    out = fg.fused_experts(*d, tw.cuda(), ids.cuda(), routed_scaling_factor=1.5, **kw)
    assert_close_moe(out, oracle(tw, ids).float() * 1.5, tol, f"{kind} T={T}")
    routed = fg.fused_moe(*d, logits.cuda(), k, True, routed_scaling_factor=1.5, **kw)
    assert_close_moe(routed, oracle(tw, ids).float() * 1.5, tol, f"{kind} T={T} with the router")
    z = fg.fused_experts(*d, tw.cuda(), ids.cuda(), no_combine=True, **kw)
    assert_close_moe(z.float().sum(1), oracle(tw, ids), tol, f"{kind} T={T} rows")
    if T > 8:
        return
    bad = ids.clone()
    bad[:, 1] = -1
    bad[0, 2] = E + 3
    if T > 1:
        bad[1] = bad[0]
    assert_close_moe(fg.fused_experts(*d, tw.cuda(), bad.cuda(), **kw), oracle(tw, bad), tol, f"{kind} T={T} dropped ids")


def _decode_call(fg, kind, T, seed, E=16, H=640, I=384, k=4):
    x, w1, w2, g = _layer(T, H, I, E, seed)
    logits = torch.randn(T, E, generator=g).cuda()
    if kind == "block":
        (w1, s1), (w2, s2) = OQ.quant_weight_block128(w1), OQ.quant_weight_block128(w2)
        kw = dict(use_fp8_w8a8=True, w1_scale=s1.cuda(), w2_scale=s2.cuda(), block_shape=[128, 128])
    else:
        kw = {}
    d = [x.cuda(), w1.cuda(), w2.cuda()]
    return lambda: fg.fused_moe(*d, logits, k, True, **kw)


@pytest.mark.parametrize("ctas", [1, 2, 29, 147])
@pytest.mark.parametrize("T", [1, 5, 8])
@pytest.mark.parametrize("kind", ["bf16", "block"])
def test_decode_layer_needs_no_cta_that_has_not_started(fg, kind, T, ctas):
    """The decode kernel's CTAs wait on one another.  Launched with fewer CTAs than it has shares of work, those that run take
    all shares, as they do while another stream holds the other SMs: the call ends and the bits are the same."""
    from flaggems_sglang_b200 import _C

    call = _decode_call(fg, kind, T, 90 + T)
    ref = call()
    _C.check(_C.lib().fmoe_debug_decode_ctas(ctas))
    out = call()
    assert torch.equal(out, ref) and torch.equal(call(), ref)


@pytest.mark.parametrize("ctas", [0, 3])
def test_decode_layer_without_an_active_expert(fg, ctas):
    """No slot has an expert: every share of the work is empty, the sums are zero."""
    from flaggems_sglang_b200 import _C

    x, w1, w2, _ = _layer(3, 256, 128, 4, 1)
    _C.check(_C.lib().fmoe_debug_decode_ctas(ctas))
    out = fg.fused_experts(x.cuda(), w1.cuda(), w2.cuda(), torch.ones(3, 2, device="cuda"), torch.full((3, 2), -1, dtype=torch.int32, device="cuda"))
    assert not out.any()


@pytest.mark.parametrize("kind", ["bf16", "block"])
def test_decode_layers_on_streams_of_two_priorities(fg, kind):
    calls = [_decode_call(fg, kind, T, 110 + T, E=32, H=1024, I=1024) for T in (1, 8)]
    refs = [c() for c in calls]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(priority=p) for p in (0, -1)]
    outs = [[], []]
    for _ in range(60):
        for i, st in enumerate(streams):
            with torch.cuda.stream(st):
                outs[i].append(calls[i]())
    torch.cuda.synchronize()
    assert all(torch.equal(o, refs[i]) for i in range(2) for o in outs[i])


def _slices(lib, tiles, k_steps, most):
    out = (ctypes.c_int64 * 5)()
    assert lib.fmoe_debug_tail_plan(tiles, k_steps, most, lib.fmoe_sm_count() // 2, 0, 0, out) == 1
    return out[4]


# one tile per expert: 16 gate/up tiles in 4 slices (32 down tiles of 8 K steps: not cut), 8 down tiles in 8 slices of 8 K steps
# (64 gate/up tiles: not cut)
@pytest.mark.parametrize("E,H,I,k", [(4, 2048, 512, 2), (2, 1024, 4096, 1)])
@pytest.mark.parametrize("T", [30, 300])
@pytest.mark.parametrize("kind", ["bf16", "n_major", "bias", "channel"])
def test_tail_split_is_finished_by_the_last_to_arrive(fg, kind, T, E, H, I, k):
    """Tiles of a part-filled last round are cut along K; the worker that arrives last adds the partials in slice order, so
    the bits do not depend on which one that is, nor on calls on a stream of another priority beside it."""
    from flaggems_sglang_b200 import _C

    step = 128 if kind == "channel" else 64  # channels of a K step
    slices = _slices(_C.lib(), E * (I // 128), H // step, 4), _slices(_C.lib(), E * (H // 256), I // step, 8)
    assert slices == ((4 // (step // 64), 1) if E == 4 else (1, 8 // (step // 64)))
    x, w1, w2, g = _layer(T, H, I, E, 130 + T)
    tw, ids = OR.softmax_topk(torch.randn(T, E, generator=g), k, True)
    idx = torch.linspace(0, T - 1, 48).long().unique()
    d, kw = [x.cuda(), w1.cuda(), w2.cuda()], dict(variant="tcgen05")
    ref = OE.fused_experts(x[idx], w1, w2, tw[idx], ids[idx])
    if kind == "n_major":
        d[1:], kw = [w.transpose(1, 2).contiguous() for w in d[1:]], dict(weights_n_major=True)
    elif kind == "bias":
        b1, b2 = torch.randn(E, 2 * I, generator=g), torch.randn(E, H, generator=g)
        kw.update(b1=b1.cuda(), b2=b2.cuda(), activation="swiglu_oai", gemm1_clamp_limit=7.0)
        ref = OE.fused_experts_with_bias(x[idx], w1, b1, w2, b2, tw[idx], ids[idx], limit=7.0)
    elif kind == "channel":
        (w1q, s1), (w2q, s2) = OQ.quant_weight_per_channel(w1), OQ.quant_weight_per_channel(w2)
        d[1:], kw = [w1q.cuda(), w2q.cuda()], dict(use_fp8_w8a8=True, per_channel_quant=True, w1_scale=s1.cuda(), w2_scale=s2.cuda())
        ref = OE.fused_experts_fp8_per_channel(x[idx], w1q, s1, w2q, s2, tw[idx], ids[idx])
    twd, idd = tw.cuda(), ids.cuda()
    call = lambda: fg.fused_experts(*d, twd, idd, **kw)  # noqa: E731
    out = call()
    assert_close_moe(out[idx.cuda()], ref, "fp8" if kind == "channel" else "bf16", f"tail split {kind} T={T}")
    decode = _decode_call(fg, "bf16", 8, 5, E=32, H=1024, I=1024)
    dref = decode()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(priority=p) for p in (0, -1, 0)]
    outs = []
    for _ in range(30):
        for st, fn, want in zip(streams, (call, call, decode), (out, out, dref)):
            with torch.cuda.stream(st):
                outs.append((fn(), want))
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o, want in outs)


@pytest.mark.parametrize("E", [1, 8, 255, 257])
@pytest.mark.parametrize("numel", [1, 127, 128, 129, 4097, 16383, 16384, 16385])
def test_align_at_chunk_edges(fg, numel, E):
    g = torch.Generator().manual_seed(numel + E)
    ids = torch.randint(-1, E + 1, (numel, 1), generator=g, dtype=torch.int32)
    s, e, n = fg.moe_align_block_size(ids.cuda(), 64, E)
    os_, oe, on = OR.moe_align_block_size(ids, 64, E)
    np.testing.assert_array_equal(n.cpu().numpy(), on)
    np.testing.assert_array_equal(s.cpu().numpy(), os_)
    np.testing.assert_array_equal(e.cpu().numpy(), oe)


@pytest.mark.parametrize("kind,T,names", [("bf16", 5, ["decode_layer"]), ("block", 5, ["decode_layer"]),
                                          ("block", 12, ["gemm1_fp8_tcgen05", "gemm2_fp8_tcgen05"]), ("bf16", 12, ["gemm1_stream", "gemm2_stream"])])
def test_stages_are_those_of_the_call(fg, kind, T, names):
    """With stage events on, the kernel family is the one that the same call takes without them."""
    import importlib

    FM = importlib.import_module("flaggems_sglang_b200.ops.fused_moe")
    call = _decode_call(fg, kind, T, 150)
    ref = call()
    FM.STAGE_EVENTS = []
    try:
        out = call()
        seen = [n for n, _, _ in FM.STAGE_EVENTS if n.startswith(("gemm", "decode"))]
    finally:
        FM.STAGE_EVENTS = None
    assert seen == names
    assert_close_moe(out, ref.cpu(), "fp8" if kind == "block" else "bf16", f"stages {kind} T={T}")


@pytest.mark.parametrize("kind,T,launches", [("bf16", 5, 2), ("block", 5, 2), ("bf16", 12, 5), ("bf16", 200, 6), ("block", 12, 7)])
def test_launches_are_counted(fg, kind, T, launches):
    """Decode: prepare and layer.  Otherwise router, block list, two GEMMs, sum, and the passes over rows in between."""
    from flaggems_sglang_b200 import _C

    call = _decode_call(fg, kind, T, 160)
    _C.lib().fmoe_debug_launches()
    call()
    assert _C.lib().fmoe_debug_launches() == launches and _C.lib().fmoe_debug_launches() == 0


@pytest.mark.parametrize("T", [1, 8, 9, 85, 86, 100, 682, 683, 2049])
def test_sorted_routing_equals_routing_by_slot(fg, T):
    """The routing triple goes to the kernels as it is; the results are those of the same routing by slot."""
    E, H, I, k = 24, 256, 192, 3
    x, w1, w2, g = _layer(T, H, I, E, 50 + T)
    logits = torch.randn(T, E, generator=g)
    tw, ids = OR.softmax_topk(logits, k, True)
    tw, ids = tw.cuda(), ids.cuda()
    rd, gi, si = fg.standard_topk_to_routing(tw, ids, E)
    ids2, perm = torch.sort(ids, dim=1)  # the triple's slots hold a token's experts in ascending order
    tw2 = torch.gather(tw, 1, perm)
    d = [x.cuda(), w1.cuda(), w2.cuda()]
    views = [d[1].transpose(1, 2), d[2].transpose(1, 2)]
    assert torch.equal(fg.triton_kernel_fused_experts(d[0], *views, rd, gi, si), fg.fused_experts(*d, tw2, ids2))
    nm = [v.contiguous() for v in views]
    assert torch.equal(fg.triton_kernel_fused_experts(d[0], *nm, rd, gi, si),
                       fg.fused_experts(d[0], *nm, tw2, ids2, weights_n_major=True))
    rows = fg.triton_kernel_fused_experts(d[0], *nm, rd, gi, None)
    ref = fg.fused_experts(d[0], *nm, tw2, ids2, weights_n_major=True, no_combine=True).view(T * k, H)[gi.src_indx.long()]
    assert torch.equal(rows, ref)


# 3 slots per token: both sides of 256 and 2048 slots, where a cluster and then two kernels make the block list
@pytest.mark.parametrize("T", [2, 30, 85, 86, 682, 683, 3000])
@pytest.mark.parametrize("fault", ["slot", "duplicate", "hist_over", "hist_negative", "hist_short"])
def test_inconsistent_triple_stays_inside_its_buffers(fg, fault, T):
    """Entries of a routing triple that only the device sees: the workspace is filled with words that would be addresses if a
    kernel took one for a position, and lies between guard bytes.  Tokens whose slots are all named once keep their rows."""
    from flaggems_sglang_b200 import _C

    E, H, I, k = 24, 256, 192, 3
    x, w1, w2, g = _layer(T, H, I, E, 70 + T)
    tw, ids = OR.softmax_topk(torch.randn(T, E, generator=g), k, True)
    xd, w1d, w2d = x.cuda(), w1.cuda(), w2.cuda()
    rd, gi, si = fg.standard_topk_to_routing(tw.cuda(), ids.cuda(), E)
    good = fg.triton_kernel_fused_experts(xd, w1d.transpose(1, 2), w2d.transpose(1, 2), rd, gi, si)
    slot_of, hist, gate = gi.src_indx.clone(), rd.expt_hist.clone(), rd.gate_scal.contiguous()
    numel, hit = T * k, torch.zeros(T, dtype=torch.bool)
    where = [0, numel // 2, numel - 1]
    if fault == "slot":
        for p, bad in zip(where, (-7, numel, 2**31 - 1)):
            hit[int(slot_of[p]) // k] = True
            slot_of[p] = bad
    elif fault == "duplicate":
        for p in where[1:]:
            hit[int(slot_of[p]) // k] = hit[int(slot_of[0]) // k] = True
            slot_of[p] = slot_of[0]
    elif fault == "hist_over":  # the last experts run past the positions: their rows are clipped
        hist[E - 1] += 2**30
    elif fault == "hist_negative":
        hit[:] = True  # every later expert's rows move
        hist[1] -= 2**31 - 1 - int(hist[1])
    else:
        cut = int(hist[hist.nonzero()[-1, 0]])
        hist[hist.nonzero()[-1, 0]] = 0
        hit[(slot_of[numel - cut:] // k).long().cpu()] = True
    lib, out = _C.lib(), torch.empty_like(xd)
    a = _C.FusedArgs(dtype=_C.BF16, num_experts=E, top_k=k, T=T, H=H, I=I, routed_scaling_factor=1.0, hidden=xd.data_ptr(),
                     w1=w1d.data_ptr(), w2=w2d.data_ptr(), out=out.data_ptr())
    need = lib.fmoe_fused_experts_sorted_workspace_bytes(a)
    guard = 1 << 20
    area = torch.full(((need + 2 * guard) // 4 + 64,), 0x3F000000, dtype=torch.int32, device="cuda")
    start = -(-(area.data_ptr() + guard) // 256) * 256
    a.workspace, a.workspace_bytes = start, need
    before = [t.clone() for t in (xd, w1d, w2d)]
    _C.check(lib.fmoe_fused_experts_sorted(a, slot_of.data_ptr(), hist.data_ptr(), gate.data_ptr(), _C.stream_ptr()))
    torch.cuda.synchronize()
    lo = (start - area.data_ptr()) // 4
    assert bool((area[:lo] == 0x3F000000).all()) and bool((area[lo + -(-need // 4):] == 0x3F000000).all())
    assert all(torch.equal(u, v) for u, v in zip(before, (xd, w1d, w2d)))
    assert torch.equal(out[~hit.cuda()], good[~hit.cuda()])
    if fault in ("slot", "hist_over", "hist_negative"):
        with pytest.raises(_C.FmoeError, match="0xB00" if fault == "slot" else "0xB01"):
            _C.check_device_status()


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 9])
def test_combine_slot_counts(fg, k):
    """moe_sum issues the loads of up to 2 or 4 slots before the first is added."""
    z = torch.randn(37, k, 264, generator=torch.Generator().manual_seed(k))
    for dt in (torch.bfloat16, torch.float32):
        out = torch.empty(37, 264, dtype=dt, device="cuda")
        fg.moe_sum(z.to(dt).cuda(), out)
        assert torch.equal(out.cpu(), OE.moe_sum(z.to(dt)).to(dt))


@pytest.mark.parametrize("T", [2, 3, 8])
def test_e4m3_layer_around_the_decode_line(fg, T):
    """Short down rows: two tokens take the decode kernels, three the CTA-pair GEMMs, in every form of the call.  Eight need more
    than the allocation-free entry holds for the pairs: it keeps the decode kernels."""
    from flaggems_sglang_b200 import _C

    E, H, I, k = 64, 7168, 256, 8
    x, w1, w2, g = _layer(T, H, I, E, 30 + T)
    logits = torch.randn(T, E, generator=g)
    tw, ids = OR.softmax_topk(logits, k, True)
    (w1q, s1), (w2q, s2) = OQ.quant_weight_block128(w1), OQ.quant_weight_block128(w2)
    d = [x.cuda(), w1q.cuda(), w2q.cuda()]
    s1d, s2d = s1.cuda(), s2.cuda()
    kw = dict(use_fp8_w8a8=True, w1_scale=s1d, w2_scale=s2d, block_shape=[128, 128])
    ref = OE.fused_experts_fp8(x, w1q, s1, w2q, s2, tw, ids)
    twd, idd = tw.cuda(), ids.cuda()
    assert_close_moe(fg.fused_experts(*d, twd, idd, **kw), ref, "fp8", f"T={T}")
    assert_close_moe(fg.fused_moe(*d, logits.cuda(), k, True, routed_scaling_factor=1.5, **kw), ref.float() * 1.5, "fp8", f"T={T} router")
    rows = fg.fused_experts(*d, twd, idd, no_combine=True, **kw)
    assert_close_moe(rows.float().sum(1), ref, "fp8", f"T={T} rows")
    first = [fg.fused_experts(*d, twd, idd, apply_router_weight_on_input=True, variant=v, **kw) for v in (None, "stream")]
    assert_close_moe(first[0], first[1].cpu(), "fp8", f"T={T} weight first")
    local = torch.arange(E, dtype=torch.int32)
    local[::2] = -1
    kept = OE.fused_experts_fp8(x, w1q, s1, w2q, s2, torch.where(ids % 2 == 1, tw, torch.zeros(())), ids)
    assert_close_moe(fg.fused_experts(*d, twd, idd, expert_map=local.cuda(), **kw), kept, "fp8", f"T={T} expert map")
    out = torch.empty(T, H, dtype=torch.bfloat16, device="cuda")
    a = _C.FusedArgs(dtype=_C.E4M3, num_experts=E, top_k=k, T=T, H=H, I=I, routed_scaling_factor=1.0, hidden=d[0].data_ptr(),
                     w1=d[1].data_ptr(), w2=d[2].data_ptr(), w1_scale=s1d.data_ptr(), w2_scale=s2d.data_ptr(),
                     topk_weights=twd.data_ptr(), topk_ids=idd.data_ptr(), out=out.data_ptr())
    lib = _C.lib()
    assert (lib.fmoe_fused_experts_workspace_bytes(a) > lib.fmoe_static_scratch_bytes()) == (T == 8)
    _C.check(lib.fmoe_fused_experts_static(a, _C.stream_ptr()))
    assert_close_moe(out, ref, "fp8", f"T={T} static")


def test_static_entry_streams_what_does_not_fit(fg):
    """e4m3 layers with few rows per expert take the padded tensor-core plan; the allocation-free entry keeps the streaming
    one where only that fits its array."""
    from flaggems_sglang_b200 import _C

    E, H, I, k, T = 128, 2048, 512, 8, 16
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(T, H, generator=g, device="cuda").bfloat16()
    w1 = (torch.randn(E, 2 * I, H, generator=g, device="cuda") * 0.5).to(torch.float8_e4m3fn)
    w2 = (torch.randn(E, H, I, generator=g, device="cuda") * 0.5).to(torch.float8_e4m3fn)
    s1 = torch.rand(E, 2 * I // 128, H // 128, generator=g, device="cuda") * 0.04
    s2 = torch.rand(E, H // 128, I // 128, generator=g, device="cuda") * 0.04
    tw, ids = fg.fused_topk(x, torch.randn(T, E, generator=g, device="cuda"), k, True)
    kw = dict(use_fp8_w8a8=True, w1_scale=s1, w2_scale=s2, block_shape=[128, 128])
    ref, auto = (fg.fused_experts(x, w1, w2, tw, ids, variant=v, **kw) for v in ("stream", None))
    out = torch.empty_like(ref)
    a = _C.FusedArgs(dtype=_C.E4M3, variant=_C.VARIANTS["auto"], num_experts=E, top_k=k, T=T, H=H, I=I, routed_scaling_factor=1.0,
                     hidden=x.data_ptr(), w1=w1.data_ptr(), w2=w2.data_ptr(), w1_scale=s1.data_ptr(), w2_scale=s2.data_ptr(),
                     topk_weights=tw.data_ptr(), topk_ids=ids.data_ptr(), out=out.data_ptr())
    lib = _C.lib()
    assert lib.fmoe_fused_experts_workspace_bytes(a) > lib.fmoe_static_scratch_bytes()
    _C.check(lib.fmoe_fused_experts_static(a, _C.stream_ptr()))
    assert torch.equal(out, ref)
    assert_close_moe(auto, ref.cpu(), "fp8", "auto against stream")


@pytest.mark.parametrize("entry", ["experts", "moe", "sorted"])
@pytest.mark.parametrize("kind,T,E,H,I,limit", [("block", 3, 64, 2048 + 7168, 256, 1 << 20), ("bf16", 24, 64, 1280, 768, 1 << 22)])
def test_workspace_that_holds_only_the_smaller_kernels(fg, entry, kind, T, E, H, I, limit):
    """The C entries with less workspace than the fastest kernels need: the decode or the streaming kernels run in it, nothing
    outside it is written."""
    from flaggems_sglang_b200 import _C

    k = 8
    x, w1, w2, g = _layer(T, H, I, E, 40 + T)
    logits = torch.randn(T, E, generator=g)
    tw, ids = OR.softmax_topk(logits, k, True)
    idx = torch.arange(0, T, 8)
    if kind == "block":
        (w1, s1), (w2, s2) = OQ.quant_weight_block128(w1), OQ.quant_weight_block128(w2)
        ref = OE.fused_experts_fp8(x[idx], w1, s1, w2, s2, tw[idx], ids[idx])
        scales = s1.cuda(), s2.cuda()
    else:
        ref, scales = OE.fused_experts(x[idx], w1, w2, tw[idx], ids[idx]), (None, None)
    lib, d = _C.lib(), [x.cuda(), w1.cuda(), w2.cuda(), tw.cuda(), ids.cuda(), logits.cuda()]
    out = torch.full((T, H), float("nan"), dtype=torch.bfloat16, device="cuda")
    a = _C.FusedArgs(dtype=_C.E4M3 if kind == "block" else _C.BF16, num_experts=E, top_k=k, T=T, H=H, I=I, routed_scaling_factor=1.0,
                     hidden=d[0].data_ptr(), w1=d[1].data_ptr(), w2=d[2].data_ptr(), w1_scale=_C.ptr(scales[0]),
                     w2_scale=_C.ptr(scales[1]), topk_weights=d[3].data_ptr(), topk_ids=d[4].data_ptr(), out=out.data_ptr())
    assert lib.fmoe_fused_experts_workspace_bytes(a) > limit
    area = torch.full((limit + 512 + 4096,), 0x5A, dtype=torch.uint8, device="cuda")
    start = -(-(area.data_ptr() + 2048) // 256) * 256
    a.workspace, a.workspace_bytes = start, limit
    st = _C.stream_ptr()
    if entry == "experts":
        _C.check(lib.fmoe_fused_experts(a, st))
    elif entry == "moe":
        _C.check(lib.fmoe_fused_moe(a, _C.RouteArgs(logits=d[5].data_ptr(), grouped=0, renormalize=1, n_group=1, topk_group=1), st))
    else:
        rd, gi, _ = fg.standard_topk_to_routing(d[3], d[4], E)
        slot_of, hist, gate = (v.contiguous() for v in (gi.src_indx, rd.expt_hist, rd.gate_scal))
        _C.check(lib.fmoe_fused_experts_sorted(a, slot_of.data_ptr(), hist.data_ptr(), gate.data_ptr(), st))
    torch.cuda.synchronize()
    lo = start - area.data_ptr()
    assert bool((area[:lo] == 0x5A).all()) and bool((area[lo + limit:] == 0x5A).all())
    assert_close_moe(out[idx.cuda()], ref, "fp8" if kind == "block" else "bf16", f"{entry} {kind} small workspace")


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("kind", ["bf16", "n_major", "channel"])
def test_units_by_ticket_are_those_dealt(fg, kind, gated):
    """Long launches of the CTA-pair GEMM take their units by ticket.  Some 70 (e4m3: 140) a worker, so that the list's places are
    used again, and tiles that are too short along K to be cut: the bits are those of units dealt round-robin, which a call without
    scratch keeps.  Beside another stream's calls too, when workers start late."""
    from flaggems_sglang_b200 import _C
    from flaggems_sglang_b200.ops.fused_moe import _gemm_args

    rows = [1, 256, 257, 900, 0, 513, 64, 511] * 3
    E, numel, k = len(rows), sum(rows), 768
    e4m3 = kind == "channel"
    steps, w_tiles = k * (1 if e4m3 else 2) // 128, 248 if e4m3 else 124
    n, lib = w_tiles * (128 if gated else 256), _C.lib()
    assert (numel // 256 + E // 2) * w_tiles * steps >= 800 * (lib.fmoe_sm_count() // 2) and steps < 16
    g = torch.Generator(device="cuda").manual_seed(5)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(rows)).to(torch.int32).view(-1, 1).cuda()
    sorted_ids, expert_ids, num_post = fg.moe_align_block_size(ids, 128, E)
    cap = sorted_ids.numel()
    dt, w_rows = torch.float8_e4m3fn if e4m3 else torch.bfloat16, (2 if gated else 1) * n
    a = torch.randn(cap, k, generator=g, device="cuda").to(dt)
    w = torch.empty(E, *((k, w_rows) if kind == "n_major" else (w_rows, k)), dtype=dt, device="cuda")
    for e in range(E):
        w[e] = (torch.randn(*w.shape[1:], generator=g, device="cuda") * k ** -0.5).to(dt)
    scales = {}
    if e4m3:
        s = torch.rand(cap, generator=g, device="cuda"), torch.rand(E, w_rows, generator=g, device="cuda")
        scales = dict(a_scale=s[0].data_ptr(), w_scale=s[1].data_ptr(), scale_mode=_C.SCALE_CHANNEL)
    split_ws = torch.empty(int(lib.fmoe_gemm_split_workspace_bytes()), dtype=torch.uint8, device="cuda")

    def call(tickets):
        out = torch.zeros(cap if gated else numel, n, dtype=torch.bfloat16, device="cuda")
        ws = dict(split_ws=split_ws.data_ptr(), split_ws_bytes=split_ws.numel()) if tickets else {}
        args = _gemm_args(variant=_C.VARIANTS["tcgen05"], activation=0, num_experts=E, top_k=1, block_size=128, numel=numel,
                          sorted_cap=cap, max_blocks=cap // 128, sorted_token_ids=sorted_ids.data_ptr(),
                          expert_ids=expert_ids.data_ptr(), num_tokens_post_padded=num_post.data_ptr(),
                          dtype=_C.E4M3 if e4m3 else _C.BF16, out_dtype=_C.BF16, n=n, k=k, a_rows=cap, a=a.data_ptr(),
                          w=w.data_ptr(), out=out.data_ptr(), w_layout=_C.W_N_MAJOR if kind == "n_major" else _C.W_K_MAJOR,
                          **scales, **ws)
        _C.check((lib.fmoe_gemm1_silu if gated else lib.fmoe_gemm2)(args, _C.stream_ptr()))
        return out

    ref = call(False)
    assert float(ref.float().abs().sum()) > 0
    other = _decode_call(fg, "bf16", 8, 5, E=32, H=1024, I=1024)
    other()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(priority=p) for p in (0, -1)]
    outs = []
    for _ in range(3):
        with torch.cuda.stream(streams[1]):
            for _ in range(8):
                other()
        with torch.cuda.stream(streams[0]):
            outs.append(call(True))
    torch.cuda.synchronize()
    assert all(torch.equal(o, ref) for o in outs)


# the gate/up GEMM (H = 32 K steps), then the down GEMM (I = 126 K steps) by ticket with the tiles of its last round cut along K
@pytest.mark.parametrize("H,I,gated", [(2048, 14336, True), (7168, 8064, False)])
@pytest.mark.parametrize("kind", ["bf16", "n_major", "channel"])
def test_units_by_ticket_with_a_cut_last_round(fg, kind, H, I, gated):
    from flaggems_sglang_b200 import _C

    lib, E, T, step = _C.lib(), 2, 4096, 64
    if kind == "channel":
        H, I, step = (2 * H, I, 128) if gated else (H, 2 * I, 128)
    steps, w_tiles = (H // step, I // 128) if gated else (I // step, H // 256)
    assert (T // 256 + E // 2) * w_tiles * steps >= 800 * (lib.fmoe_sm_count() // 2)
    slices = (ctypes.c_int64 * 5)()
    tiles, workers = T // 256 * w_tiles, lib.fmoe_sm_count() // 2
    assert lib.fmoe_debug_tail_plan(tiles, steps, 4 if gated else 8, workers, 0, -(-tiles // workers) - 1, slices) == 1 and slices[4] > 1
    gd = torch.Generator(device="cuda").manual_seed(18)
    w1 = torch.stack([(torch.randn(2 * I, H, generator=gd, device="cuda") * H ** -0.5).bfloat16() for _ in range(E)])
    w2 = torch.stack([(torch.randn(H, I, generator=gd, device="cuda") * I ** -0.5).bfloat16() for _ in range(E)])
    g = torch.Generator().manual_seed(17)
    x, tw = torch.randn(T, H, generator=g).bfloat16(), torch.rand(T, 1, generator=g) + 0.5
    ids = torch.arange(E).repeat(T // E).to(torch.int32).view(T, 1)
    idx = torch.linspace(0, T - 1, 8).long()
    d, kw = [x.cuda(), w1, w2], dict(variant="tcgen05")
    c1, c2 = w1.cpu(), w2.cpu()
    if kind == "n_major":
        d[1:], kw = [w.transpose(1, 2).contiguous() for w in d[1:]], dict(weights_n_major=True)
    if kind == "channel":
        (q1, s1), (q2, s2) = OQ.quant_weight_per_channel(c1), OQ.quant_weight_per_channel(c2)
        ref = OE.fused_experts_fp8_per_channel(x[idx], q1, s1, q2, s2, tw[idx], ids[idx])
        d[1:], kw = [q1.cuda(), q2.cuda()], dict(use_fp8_w8a8=True, per_channel_quant=True, w1_scale=s1.cuda(), w2_scale=s2.cuda())
    else:
        ref = OE.fused_experts(x[idx], c1, c2, tw[idx], ids[idx])
    outs = [fg.fused_experts(*d, tw.cuda(), ids.cuda(), **kw) for _ in range(3)]
    assert_close_moe(outs[0][idx.cuda()], ref, "fp8" if kind == "channel" else "bf16", f"tickets {kind} H={H}")
    assert all(torch.equal(o, outs[0]) for o in outs)


def test_wait_profile_has_a_word_for_each_producer():
    """FMOE_TC_PROFILE: both TMA warps of a CTA leave their waits, in words of their own."""
    code = """
import ctypes, torch
import flaggems_sglang_b200 as fg
from flaggems_sglang_b200 import _C
E, H, I, T = 8, 2048, 2048, 2048
w1, w2 = (torch.randn(E, *s, device="cuda").mul_(0.02).bfloat16() for s in ((2 * I, H), (H, I)))
x, logits = torch.randn(T, H, device="cuda").bfloat16(), torch.randn(T, E, device="cuda")
fg.fused_moe(x, w1, w2, logits, 2, True, variant="tcgen05")
_C.check_device_status()
n = _C.lib().fmoe_sm_count() // 2 * 2
buf = (ctypes.c_int64 * (n * 8))()
_C.check(_C.lib().fmoe_debug_wait_profile(_C.VARIANTS["tcgen05"], buf, n * 8))
a = torch.tensor(list(buf)).view(n, 8)
assert bool((a[:, 3] > 0).all()) and bool((a[:, 6] > 0).all()), a[:4]
"""
    env = dict(os.environ, FMOE_TC_PROFILE="1", PYTHONPATH=os.pathsep.join(sys.path))
    subprocess.run([sys.executable, "-c", code], check=True, env=env, timeout=300)


def test_calls_in_one_workspace_whose_routing_changes(tmp_path):
    """The CTA-pair GEMMs read the expert table and weights, and take tickets, ahead of their wait for the kernel before.  Calls of
    one workspace follow one another without a synchronisation, each with another routing (few hot experts, other ones, all, a
    different number of tokens), so that a table or a counter of the call before would give other rows: the bits are those of calls
    that are waited for, with programmatic launches and with plain ones."""
    code = """
import sys, torch
import flaggems_sglang_b200 as fg
from flaggems_sglang_b200 import _C
lib, st = _C.lib(), _C.stream_ptr()
g = torch.Generator(device="cuda").manual_seed(1)
rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
E, k, outs = 16, 4, []
for kind, H, I, sizes in (("bf16", 1024, 1024, (700, 301)), ("bf16", 4096, 7168, (2048, 1500)), ("n_major", 1024, 1024, (700, 301)),
                          ("channel", 1024, 1024, (700, 301)), ("block", 1024, 1024, (700, 301)), ("block", 1024, 512, (90, 40))):
    w1, w2 = rand(E, 2 * I, H) * H ** -0.5, rand(E, H, I) * I ** -0.5
    s1 = s2 = None
    if kind in ("block", "channel"):
        quant = fg.quant_weight_block128 if kind == "block" else fg.quant_weight_per_channel
        (w1, s1), (w2, s2) = (tuple(torch.stack(v) for v in zip(*(quant(e) for e in w))) for w in (w1, w2))
    else:
        w1, w2 = w1.bfloat16(), w2.bfloat16()
    if kind == "n_major":
        w1, w2 = w1.transpose(1, 2).contiguous(), w2.transpose(1, 2).contiguous()
    calls = []
    for i in range(8):
        T = sizes[i % 2]
        logits = rand(T, E)
        if i % 4 != 3:
            logits[:, (5 * i + torch.arange(6, device="cuda")) % E] += 4.0  # six hot experts, others in each call
        x, out = rand(T, H).bfloat16(), torch.empty(T, H, dtype=torch.bfloat16, device="cuda")
        a = _C.FusedArgs(dtype=_C.E4M3 if s1 is not None else _C.BF16, variant=_C.VARIANTS["tcgen05"], num_experts=E, top_k=k, T=T, H=H, I=I,
                         routed_scaling_factor=1.0, hidden=x.data_ptr(), w1=w1.data_ptr(), w2=w2.data_ptr(), w1_scale=_C.ptr(s1),
                         w2_scale=_C.ptr(s2), out=out.data_ptr(), w_layout=_C.W_N_MAJOR if kind == "n_major" else _C.W_K_MAJOR,
                         scale_mode=_C.SCALE_CHANNEL if kind == "channel" else _C.SCALE_BLOCK128)
        calls.append((a, _C.RouteArgs(logits=logits.data_ptr(), grouped=0, renormalize=1, n_group=1, topk_group=1), out, (x, logits)))
    need = max(lib.fmoe_fused_moe_workspace_bytes(a, r) for a, r, _, _ in calls)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    refs = []
    for a, r, out, _ in calls:
        a.workspace, a.workspace_bytes = ws.data_ptr(), need
        _C.check(lib.fmoe_fused_moe(a, r, st))
        torch.cuda.synchronize()
        refs.append(out.clone())
        assert float(refs[-1].float().abs().sum()) > 0
    for _ in range(12):
        for _, _, out, _ in calls:
            out.fill_(float("nan"))
        torch.cuda._sleep(2000000)  # the calls queue up behind it
        for a, r, _, _ in calls:
            _C.check(lib.fmoe_fused_moe(a, r, st))
        torch.cuda.synchronize()
        assert all(torch.equal(out, ref) for (_, _, out, _), ref in zip(calls, refs)), (kind, H, I)
    outs += [r.cpu() for r in refs]
fg._C.check_device_status()
torch.save(outs, sys.argv[1])
"""
    outs = []
    for pdl in ("1", "0"):
        path = str(tmp_path / f"out{pdl}.pt")
        env = dict(os.environ, FMOE_PDL=pdl, PYTHONPATH=os.pathsep.join(sys.path))
        subprocess.run([sys.executable, "-c", code, path], check=True, env=env, timeout=300)
        outs.append(torch.load(path))
    assert all(torch.equal(a, b) for a, b in zip(*outs))
