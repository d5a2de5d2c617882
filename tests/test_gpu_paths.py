"""Edges of the dispatch and of the kernels' partitions, against the CPU oracle on the same seeded inputs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from berth_b200 import Codebook, OutDtype, kernels, moe, synth   # noqa: E402
from tests.gpu_util import assert_close, dev, run_linear   # noqa: E402
from tests.test_gpu_parity import test_rms_norm_bit_exact as rms_norm_bit_exact   # noqa: E402


def test_integer_path_one_hot_blocks(oracle):
    """An input with one element per 128-block rotates to blocks whose values are all alike; a block's product with the
    weights' byte sums (128 x 510 x 32512 on average) then lies around 2^31."""
    K, N, bits, cb = 512, 2048, 4, 2
    w = synth.linear_weights(1234, "onehot", K, N, bits)
    x = np.zeros((1, K), np.float16)
    x[0, ::128] = [1.0, -2.0, 0.5, 3.0]
    c, _ = run_linear(x, w, bits, cb, True)
    assert "k_exl3_gemv_i8" in kernels.last_launch()
    assert_close(c, oracle.linear_f64(x, w["trellis"], w["suh"], w["svh"], K, N, bits, cb), "one-hot blocks")


@pytest.mark.parametrize("m,bits", [(1, 4), (1, 5), (4, 4), (4, 5)])
def test_integer_path_sums_are_rounded_not_cut(oracle, m, bits):
    """A row that rotates to two non-zero values, quantised to 32512 and 13, so that the integer sum of a column is known:
    32512 u1 + 13 u2 (u the weights' byte sums).  The first output of a band adds its 128 columns: rounding errors of a sum (half a
    unit) average out over 96 bands, to about 12 / sqrt(96) units by the fp32 roundings behind them, a low bit that is always
    dropped (half a unit of every column) does not: 64."""
    f, N, i0, i1 = np.float32, 128 * 96, 5, 77
    w = synth.linear_weights(1234, f"round{bits}", 128, N, bits)
    sign = np.array([[(-1) ** bin(i & j).count("1") for j in range(128)] for i in (i0, i1)])
    same = sign[0] == sign[1]
    x = np.where(same, 1301, 1413) / 128 * sign[0]                       # times suh: (32512 s0 + 13 s1) / 128
    w["suh"], w["svh"] = np.where(same, 25, 23).astype(np.float16), np.ones(N, np.float16)
    u = np.rint((oracle.reconstruct(w["trellis"], 128, N, bits, 2).view(np.float16).reshape(128, N).astype(np.float64) + 10.3828125) / 0.00676727294921875) - 1024
    total = 32512 * u[i0] + 13 * u[i1]
    scale = f(f(32512) * f(0.088388347648)) * f(1 / 32512)
    constant = f(f(-3.453125) * f(scale * f(32525)))
    exp = (0.00676727294921875 * np.float64(scale) * total + np.float64(constant)).reshape(96, 128).sum(1) * 0.088388347648
    c, _ = run_linear(np.tile(x, (m, 1)).astype(np.float16), w, bits, 2, True)
    assert "k_exl3_gemv_i8" in kernels.last_launch()
    for row in c:
        units = (row[::128] - exp) / (0.00676727294921875 * np.float64(scale) * 0.088388347648)
        assert abs(units.mean()) < 8 and np.abs(units).max() < 200, (units.mean(), np.abs(units).max())


@pytest.mark.parametrize("bits", [3, 4, 5, 6])
@pytest.mark.parametrize("K,N", [(128, 128 * 301), (384, 256 * 160 + 128)])
def test_integer_path_several_band_groups_per_cta(oracle, K, N, bits):
    """So many columns that a CTA holds whole band groups and meets every 128-block of the row again and again."""
    w = synth.linear_weights(1234, f"wide{K}{bits}", K, N, bits)
    x = synth.activations(1234, f"wide{K}.x", 1, K)
    c, _ = run_linear(x, w, bits, 2, True)
    assert "k_exl3_gemv_i8" in kernels.last_launch() and "fused" in kernels.last_launch()
    assert_close(c, oracle.linear_f64(x, w["trellis"], w["suh"], w["svh"], K, N, bits, 2), "wide")
    assert kernels.device_status(torch.cuda.current_device()) == 0

@pytest.mark.parametrize("m,K,N,bits,here", [(m, K, N, bits, m in where) for K, N, bits, where in [
    (5120, 1024, 4, (2,)), (5120, 1024, 5, (2, 3, 4)), (2176, 3072, 5, (2, 3, 4)), (1024, 128 * 80, 6, (3, 4)), (896, 8192, 6, ()),
    (128, 128 * 301, 6, (2, 3, 4)), (384, 128 * 301, 5, (2, 3, 4)), (2048, 128 * 100, 8, (3, 4)), (1152, 640, 3, (2,)), (1024, 640, 3, (2, 3, 4)),
    (256, 128 * 301, 4, (2, 3, 4)), (2048, 128 * 301, 4, (2,)), (2176, 128 * 301, 4, ()), (3584, 128 * 130, 5, (3,)), (2048, 6144, 3, (3,)),
    (2048, 128 * 96, 4, (3,)), (3072, 3072, 4, ()), (3072, 6400, 3, (3,))] for m in (2, 3, 4)])
def test_integer_path_two_to_four_rows(oracle, m, K, N, bits, here):
    """Both sides of each line of the rule that picks the kernel."""
    w = synth.linear_weights(1234, f"few{K}{bits}", K, N, bits)
    x = synth.activations(1234, f"few{K}.x{m}", m, K)
    c, ah = run_linear(x, w, bits, 2, False)
    assert ("k_exl3_gemv_i8" in kernels.last_launch()) == here and ("fused" in kernels.last_launch() or not here)
    assert_close(c, oracle.linear_f64(x, w["trellis"], w["suh"], w["svh"], K, N, bits, 2), "few rows")
    assert (ah == oracle.had_r_128(x, w["suh"], True).view(np.uint16)).all()

@pytest.mark.parametrize("m,K,N,bits,here", [(2, 5120, 4096, 4, True), (3, 5120, 2048, 4, True), (3, 10240, 8192, 4, True), (3, 10240, 8192, 3, False), (4, 5120, 2048, 4, True), (4, 5120, 8192, 5, False)])
def test_integer_path_two_to_four_rows_silu(oracle, m, K, N, bits, here):
    """The down projection's rule: silu(gate) * up in the rotation, short and long ones."""
    w = synth.linear_weights(1234, f"fewsilu{K}{N}", K, N, bits)
    gate, up = (synth.activations(1234, f"fewsilu.{c}{m}", m, K) for c in "gu")
    c, ah = torch.empty((m, N), dtype=torch.float32, device="cuda"), torch.empty((m, K), dtype=torch.float16, device="cuda")
    kernels.exl3_linear_silu(dev(gate), dev(up), dev(w["trellis"]), c, dev(w["suh"]), ah, dev(w["svh"]), m, K, N, bits, Codebook(2), OutDtype.F32)
    torch.cuda.synchronize()
    assert ("k_exl3_gemv_i8" in kernels.last_launch()) == here
    x = oracle.silu_mul(gate.ravel(), up.ravel(), 0.0).view(np.float16).reshape(m, K)
    assert_close(c.cpu().numpy(), oracle.linear_f64(x, w["trellis"], w["suh"], w["svh"], K, N, bits, 2), "silu")

@pytest.mark.parametrize("m,N,inside", [(2, 128 * 720, True), (2, 128 * 760, False), (3, 128 * 720, True), (4, 128 * 360, True), (4, 128 * 380, False)])
def test_stack_rotation_inside_or_before(oracle, m, N, inside):
    """78 and 84 blocks a CTA of two rows, 117 of three, 80 and 84 of four: rotated in the launch or by launches before it."""
    K, bits, ns = 512, 5, 2
    ws = [synth.linear_weights(1234, f"stk{N}.{i}", K, N, bits) for i in range(ns)]
    x = synth.activations(1234, f"stk.x{m}", m, K)
    tr, su, sv = (torch.stack([dev(w[k]) for w in ws]) for k in ("trellis", "suh", "svh"))
    c, ah = torch.empty((ns, m, N), dtype=torch.float32, device="cuda"), torch.empty((ns, m, K), dtype=torch.float16, device="cuda")
    kernels.exl3_linear_stack(dev(x), tr, c, su, ah, sv, ns, m, K, N, bits, Codebook(2), OutDtype.F32)
    torch.cuda.synchronize()
    assert ("fused" in kernels.last_launch()) == inside and "k_exl3_gemv_i8" in kernels.last_launch()
    for i, w in enumerate(ws):
        assert_close(c[i].cpu().numpy(), oracle.linear_f64(x, w["trellis"], w["suh"], w["svh"], K, N, bits, 2), "stack")

@pytest.mark.parametrize("T", [1, 2, 3, 4, 5, 9])
@pytest.mark.parametrize("bits,inter,shared,E", [(4, 128, 128, 32), (3, 384, 384, 64), (5, 256, 0, 32)])
def test_moe_layer_few_tokens_vs_oracle(oracle, T, bits, inter, shared, E):
    """One launch per projection (up to four tokens) and the grouped decode launches above, gate and up as one stack and
    apart, the shared expert inside the stacks, apart and absent."""
    H, k = 512, 8
    wts = synth.moe_layer_weights(1234, f"few{bits}", H, inter, E, k, bits, 2, shared_inter=shared)
    x = synth.activations(1234, f"few.x{T}", T, H)
    for pair, fuse in ((True, True), (False, False)):
        layer = moe.MoeLayer(torch.device("cuda"), wts, T, fuse_shared=fuse, pair_gate_up=pair)
        out = torch.full((T, H), float("nan"), dtype=torch.float32, device="cuda")
        idx = torch.empty((T, k), dtype=torch.int32, device="cuda")
        w = torch.empty((T, k), dtype=torch.float32, device="cuda")
        layer.forward(dev(x), out, idx, w)
        torch.cuda.synchronize()
        assert kernels.device_status(torch.cuda.current_device()) == 0
        assert ("fused,grouped" in moe.last_launch()) == (T <= 4)
        _, exp_idx, exp_w = oracle.moe_layer(wts, x)
        assert (idx.cpu().numpy() == exp_idx).all()
        assert_close(out.cpu().numpy(), oracle.moe_layer_f64(wts, x, exp_idx, exp_w), f"T={T} pair={pair}")

@pytest.mark.parametrize("T", [1, 2, 18, 19, 37, 75, 150])
@pytest.mark.parametrize("H,E", [(2048, 256), (96, 64), (1056, 512)])
def test_router_tiles_bit_exact(oracle, T, H, E):
    """Every token tile of the router (one, two, four, eight tokens per block; the row remainders of its unrolled loops)."""
    k = 8
    x, w = synth.activations(1234, f"rt.x{T}", T, H), synth.router_weight(1234, f"rt{H}", H, E)
    idx = torch.empty((T, k), dtype=torch.int32, device="cuda")
    tw = torch.empty((T, k), dtype=torch.float32, device="cuda")
    logits = torch.empty((T, E), dtype=torch.float32, device="cuda")
    moe.router_topk(dev(x), dev(w), None, idx, tw, logits, T, H, E, k)
    torch.cuda.synchronize()
    tok = next((t for t in (1, 2, 4, 8) if E // 32 * -(-T // t) <= kernels.device_sms(torch.cuda.current_device())), 8)
    assert f",{tok}> grid={E // 32}x{-(-T // tok)} " in moe.last_launch()
    exp_logits = oracle.router_logits(x, w)
    exp_idx, exp_w = oracle.router_topk(exp_logits, k)
    assert (logits.cpu().numpy().view(np.uint32) == exp_logits.view(np.uint32)).all()
    assert (idx.cpu().numpy() == exp_idx).all()
    assert np.abs(tw.cpu().numpy() - exp_w).max() <= 1e-6

@pytest.mark.parametrize("m,K,N,bits,cb,out_fp32,rows,split", [
    (33, 512, 128, 4, 2, True, 128, 1), (64, 5120, 1024, 3, 2, False, 128, 8), (97, 2176, 384, 5, 0, True, 128, 8), (129, 4096, 256, 4, 1, False, 128, 8),
    (200, 1664, 640, 6, 2, False, 128, 6), (256, 2048, 128, 8, 2, True, 128, 8), (300, 5120, 256, 1, 2, False, 128, 8), (384, 3968, 128, 4, 2, True, 128, 8),
    (421, 5120, 1024, 4, 2, False, 128, 4), (40, 128, 128, 4, 2, True, 128, 1), (40, 384, 128, 4, 2, True, 128, 1),
    (150, 2048, 1024, 4, 2, True, 256, 8), (300, 1024, 2176, 5, 2, False, 256, 3), (150, 1024, 2176, 3, 0, True, 256, 4), (300, 512, 6400, 4, 2, False, 384, 2)])
def test_prefill_split_k(oracle, m, K, N, bits, cb, out_fp32, rows, split):
    """Few bands: the tile's K is split over a cluster (up to eight CTAs, uneven shares, passes without an owner's partner, all
    three tile heights); K below four stages per CTA is not.  On a GPU of 148 SMs the split follows from the shape."""
    w = synth.linear_weights(1234, f"split{K}{bits}", K, N, bits)
    x = synth.activations(1234, f"split{K}.x", m, K)
    c, _ = run_linear(x, w, bits, cb, out_fp32, prefill=True)
    launch = kernels.prefill_lin.last_launch()
    assert "k_exl3_gemm_tc" in launch
    if kernels.device_sms(torch.cuda.current_device()) == 148:
        assert f"grid={N // 128}x{-(-m // rows)}" + (f"x{split} " if split > 1 else " ") in launch and f"tile={rows}x" in launch
    assert_close(c, oracle.linear_f64(x, w["trellis"], w["suh"], w["svh"], K, N, bits, cb), "split K")
    for _ in range(2):      # fixed order of the partial sums
        again, _ = run_linear(x, w, bits, cb, out_fp32, prefill=True)
        assert again.tobytes() == c.tobytes()
    assert kernels.device_status(torch.cuda.current_device()) == 0


@pytest.mark.parametrize("rows,K,skip", [(421, 5120, 0), (74, 128 * 128, 0), (9473, 128, 0), (3159, 384, 0), (421, 5120, 4)])
def test_rotation_of_many_rows_bit_exact(oracle, rows, K, skip):
    """Enough 128-blocks for the wide form: a last group of one block, three blocks per row, and pointers off the 16-byte
    boundary, which keep the narrow one."""
    x, w = synth.activations(1234, f"rot{K}", rows, K), synth.linear_weights(1234, f"rot{K}", K, 128, 4)
    buf = torch.zeros(rows * K + skip, dtype=torch.float16, device="cuda")
    buf[skip:] = dev(x).view(-1)
    out = torch.empty((rows, K), dtype=torch.float16, device="cuda")
    kernels.prefill_lin.had_r_128(buf[skip:], out, dev(w["suh"]), True, rows, K, False)
    torch.cuda.synchronize()
    assert ("k_had128_wide" in kernels.prefill_lin.last_launch()) == (skip == 0)
    assert (out.cpu().numpy().view(np.uint16) == oracle.had_r_128(x, w["suh"], True).view(np.uint16)).all()


@pytest.mark.parametrize("n,limit,skip", [(65536, 0.0, 0), (65536 * 16, 0.0, 0), (65536 * 16, 3.5, 0), (65536 * 16 + 2, 0.0, 0), (65536 * 16, 0.0, 2)])
def test_silu_mul_every_gate_value_bit_exact(oracle, n, limit, skip):
    """All 65536 fp16 patterns as gates (NaN and infinities among them), in the wide and the narrow form."""
    gate = np.resize(np.arange(65536, dtype=np.uint16), n).view(np.float16)
    up = synth.activations(1234, "silu.u", 1, n)[0]
    g, u = (torch.zeros(n + skip, dtype=torch.float16, device="cuda") for _ in range(2))
    g[skip:], u[skip:] = dev(gate), dev(up)
    out = torch.empty(n, dtype=torch.float16, device="cuda")
    kernels.ops.silu_mul(g[skip:], u[skip:], out, n, limit)
    torch.cuda.synchronize()
    assert ("k_silu_mul_wide" in kernels.ops.last_launch()) == (n == 65536 * 16 and skip == 0)
    got, exp = out.cpu().numpy(), oracle.silu_mul(gate, up, limit)
    nan = np.isnan(exp)
    assert (np.isnan(got) == nan).all()
    assert (got.view(np.uint16)[~nan] == exp.view(np.uint16)[~nan]).all()


def _written_by_a_slow_kernel(seed, n):
    """A buffer of n halves and a call that fills it on the stream with one row of RMSNorm: one block, which lets its successor
    start at once and writes the end of the row last."""
    x, wn = dev(synth.activations(seed, "slow.x", 1, n).astype(np.float32)), torch.zeros(n, dtype=torch.float16, device="cuda")
    y = torch.zeros(n, dtype=torch.float16, device="cuda")
    return y, lambda: kernels.ops.rms_norm(x, wn, y, 1, n, 1e-6, 1.0, 1.0, False)


@pytest.mark.parametrize("m,K,N,bits,cb,kernel", [(1, 1024, 256, 4, 2, "k_exl3_gemv_i8"), (3, 1024, 256, 5, 2, "k_exl3_gemv_i8"), (8, 1024, 256, 4, 0, "k_exl3_gemv<"),
                                                  (20, 2048, 5120, 4, 2, "splitk"), (40, 1024, 256, 4, 2, "x1x"), (40, 128, 512, 4, 2, "grid=4x1 "),
                                                  (300, 1024, 256, 5, 1, "k_exl3_gemm_tc")])
def test_output_scales_written_by_the_preceding_kernel(m, K, N, bits, cb, kernel):
    """svh is touched only after the predecessor ended, on every path: it may be the preceding kernel's output."""
    w = synth.linear_weights(1234, f"svh{K}x{N}", K, N, bits)
    x, td, sd = dev(synth.activations(1234, f"svh.x{m}", m, K)), dev(w["trellis"]), dev(w["suh"])
    slow, write = _written_by_a_slow_kernel(1234, 65536)
    svh = slow[-N:]
    c, ah = torch.empty((m, N), dtype=torch.float32, device="cuda"), torch.empty((m, K), dtype=torch.float16, device="cuda")
    linear = lambda: kernels.exl3_linear(x, td, c, sd, ah, svh, m, K, N, bits, Codebook(cb), OutDtype.F32)
    write()
    torch.cuda.synchronize()
    linear()
    ref = c.cpu().numpy()
    assert kernel in kernels.last_launch()
    for _ in range(8):
        slow.zero_()
        torch.cuda.synchronize()
        write()
        linear()
        assert (c.cpu().numpy().view(np.uint32) == ref.view(np.uint32)).all()


@pytest.mark.parametrize("m,K,N,bits,cb,guard", [(1, 1024, 256, 4, 2, True), (3, 1024, 256, 4, 2, True), (8, 1024, 256, 4, 0, True), (20, 2048, 5120, 4, 2, True),
                                                 (40, 1024, 256, 4, 2, False), (40, 1024, 256, 4, 2, True), (40, 128, 512, 4, 2, False),
                                                 (300, 1024, 256, 5, 1, False), (300, 512, 4096, 3, 2, False)])
def test_weights_written_by_the_preceding_kernel(m, K, N, bits, cb, guard):
    """The trellis as the output of the kernel that directly precedes the linear: above 32 rows at any time, on the decode
    kernels with berth_exl3_weights_streamed(1)."""
    w = synth.linear_weights(1234, f"trw{K}x{N}", K, N, bits)
    x, sd, vd = dev(synth.activations(1234, f"trw.x{m}", m, K)), dev(w["suh"]), dev(w["svh"])
    trellis, write = _written_by_a_slow_kernel(1234, K * N * bits // 16)
    c, ah = torch.empty((m, N), dtype=torch.float32, device="cuda"), torch.empty((m, K), dtype=torch.float16, device="cuda")
    linear = lambda: kernels.exl3_linear(x, trellis, c, sd, ah, vd, m, K, N, bits, Codebook(cb), OutDtype.F32)
    write()
    torch.cuda.synchronize()
    linear()
    ref = c.cpu().numpy()
    assert np.isfinite(ref).all()
    assert kernels.weights_streamed(guard) is False
    try:
        for _ in range(8):
            trellis.zero_()
            torch.cuda.synchronize()
            write()
            linear()
            assert (c.cpu().numpy().view(np.uint32) == ref.view(np.uint32)).all()
    finally:
        kernels.weights_streamed(False)


@pytest.mark.parametrize("send,local", [(6, 1), (6, 2), (9, 3), (6, 0), (2, 4), (1, 3), (4, 4), (3, 1)])
def test_peer_experts_of_more_sent_than_local_tokens(oracle, send, local):
    """berth_moe_p2p_experts takes the tokens that were sent and those of the shared expert apart: one rank that is its own peer,
    its "symmetric" buffers ordinary allocations.  The sent tokens' rows come back as the oracle's layer without a shared
    expert, the shared rows as its difference to the layer with one."""
    import ctypes as C
    from berth_b200 import _lib
    H, I, E, k, bits = 256, 128, 32, 4, 4
    l, device = _lib.lib(), torch.device("cuda", torch.cuda.current_device())
    wts = synth.moe_layer_weights(1234, "p2pn", H, I, E, k, bits, 2, shared_inter=I)
    stages = moe.GpuStages(device, wts, E, max_rows=128, max_rows_per_expert=32)
    assert stages.shared_is_stacked()
    xh = synth.activations(1234, "p2pn.x", max(send, local), H)
    x, max_rows = dev(xh), send * k + max(send, local) + 1
    z = lambda n, dt=torch.uint8: torch.zeros(n, dtype=dt, device=device)
    cnt, flags, recv, ret = z(E * 4), z(3 * 8 * 4), z(max_rows * H * 2), torch.full((send * k, H), float("nan"), dtype=torch.float16, device=device)
    ptr = lambda t: (C.c_void_p * 1)(t.data_ptr())
    send_ws, ws = z(l.berth_moe_p2p_send_workspace_bytes(send, E, k, 1)), z(l.berth_moe_p2p_experts_workspace_bytes(max_rows, E, H, I))
    idx, w, inv = z(send * k, torch.int32), z(send * k, torch.float32), z(send * k, torch.int32)
    ysh = torch.full((max(local, 1), H), float("nan"), dtype=torch.float16, device=device)
    for epoch in (1, 2):
        assert l.berth_moe_p2p_send(x.data_ptr(), send, stages.layer._keep["w_router"].data_ptr(), None, H, E, k, idx.data_ptr(), w.data_ptr(),
                                    inv.data_ptr(), 0, 1, epoch, ptr(cnt), ptr(flags), ptr(recv), max_rows, send_ws.data_ptr(), send_ws.numel(), None) == 0
        assert l.berth_moe_p2p_experts(C.byref(stages.layer.c), x.data_ptr(), local, ysh.data_ptr() if local else None, 0, 1, epoch, E, k, send,
                                       ptr(cnt), ptr(flags), ptr(recv), ptr(ret), max_rows, send * k, 8, send_ws.data_ptr(), ws.data_ptr(),
                                       ws.numel(), None) == 0, moe.last_error()
    assert ("fused,grouped" in moe.last_launch()) == (max(send, local) <= 4)
    out = stages.combine(ret, inv, w.view(send, k), None)
    torch.cuda.synchronize()
    assert kernels.device_status(device.index) == 0
    alone = dict(wts, shared_inter=0)
    _, exp_idx, exp_w = oracle.moe_layer(alone, xh)
    assert (idx.view(send, k).cpu().numpy() == exp_idx[:send]).all()
    routed = oracle.moe_layer_f64(alone, xh, exp_idx, exp_w)
    assert_close(out.cpu().numpy(), routed[:send], "routed")
    if local:
        assert_close(ysh.cpu().numpy(), (oracle.moe_layer_f64(wts, xh, exp_idx, exp_w) - routed)[:local], "shared")


@pytest.mark.parametrize("m,K,N,cb", [(40, 5120, 256, 0), (33, 5120, 1024, 2), (200, 2048, 512, 1), (421, 1024, 384, 2)])
def test_prefill_8_bits_many_stages(oracle, m, K, N, cb):
    """8 bits: seven trellis stages for four decode groups, whose phases are told apart by waiting in the MMAs' order."""
    w = synth.linear_weights(1234, f"b8{K}", K, N, 8)
    x = synth.activations(1234, f"b8{K}.x", m, K)
    exp = oracle.linear_f64(x, w["trellis"], w["suh"], w["svh"], K, N, 8, cb)
    first = None
    for _ in range(20):
        c, _ = run_linear(x, w, 8, cb, True, prefill=True)
        assert first is None or c.tobytes() == first.tobytes()
        first = c
    assert "k_exl3_gemm_tc" in kernels.prefill_lin.last_launch()
    assert_close(first, exp, "8 bits")
    assert kernels.device_status(torch.cuda.current_device()) == 0


@pytest.mark.parametrize("H,inter", [(512, 1152), (2048, 256)])
def test_moe_layer_8_bits_tensor_core_stage(oracle, H, inter):
    """The same in the grouped kernel: a long K (four decode groups) and a short one (three groups, two epilogue teams)."""
    E, k, T = 32, 8, 128
    wts = synth.moe_layer_weights(1234, "moe8", H, inter, E, k, 8, 2, shared_inter=inter)
    x = synth.activations(1234, "moe8.x", T, H)
    layer = moe.MoeLayer(torch.device("cuda"), wts, T)
    out = torch.full((T, H), float("nan"), dtype=torch.float32, device="cuda")
    idx, w = torch.empty((T, k), dtype=torch.int32, device="cuda"), torch.empty((T, k), dtype=torch.float32, device="cuda")
    for _ in range(10):
        layer.forward(dev(x), out, idx, w)
        torch.cuda.synchronize()
    assert "k_exl3_gemm_tc_grouped" in moe.last_launch()
    assert kernels.device_status(torch.cuda.current_device()) == 0
    _, exp_idx, exp_w = oracle.moe_layer(wts, x)
    assert (idx.cpu().numpy() == exp_idx).all()
    assert_close(out.cpu().numpy(), oracle.moe_layer_f64(wts, x, exp_idx, exp_w), "8 bits")


@pytest.mark.parametrize("rows,dim", [(2, 2048), (2, 2052), (1, 3000), (3, 4096), (1, 4100), (2, 6148), (3, 8192), (2, 8196), (1, 12288)])
@pytest.mark.parametrize("wbf", [True, False])
def test_rms_norm_groups_in_registers(oracle, rows, dim, wbf):
    """4, 8, 12 or 16 groups of four per thread held in registers, at the edges of each, and the loop above 8192 columns."""
    rms_norm_bit_exact(oracle, rows, dim, wbf)
