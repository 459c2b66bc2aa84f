"""Kernels whose tile is chosen by size, at the sizes where a tile, a chunk or a group ends in the middle."""
import pytest

import darknet_b200 as dn
from conftest import parity
from test_gpu_layers import conv_case, oracle_conv, run_conv

pytestmark = pytest.mark.gpu

FP32_TILES = {   # tile of the fp32 GEMM -> cases; 296 blocks of 128 x 64 (or x 32) fill an SM twice
    "large_tile_64_filters_ragged": dict(b=5, c=5, h=89, w=87, n=65, size=3),
    "large_tile_32_filters": dict(b=5, c=9, h=90, w=86, n=31, size=3, stride=1, act="linear"),
    "large_tile_1x1_odd_channels": dict(b=6, c=21, h=81, w=83, n=70, size=1),
    "small_tile_one_pixel_over": dict(b=1, c=10, h=3, w=11, n=33, size=3),
    "small_tile_stride2": dict(b=2, c=24, h=9, w=13, n=17, size=3, stride=2),
    "small_tile_1x1_one_channel_over": dict(b=1, c=17, h=5, w=7, n=18, size=1),
    "groups_off_four_channel_boundary": dict(b=2, c=36, h=9, w=10, n=38, size=3, groups=2),
    "groups_of_four_channels": dict(b=2, c=16, h=9, w=10, n=40, size=3, groups=2),
    "slab_4": dict(b=2, c=24, h=7, w=9, n=9, size=3, groups=3),
    "slab_8": dict(b=2, c=12, h=7, w=9, n=15, size=3, groups=3),
    "slab_16": dict(b=1, c=6, h=9, w=15, n=15, size=3, pad=0),
}


@pytest.mark.parametrize("name", list(FP32_TILES))
@pytest.mark.parametrize("layouts", [("nchw", "nchw"), ("nchw", "nhwc"), ("nhwc", "nhwc")])
def test_fp32_gemm_tiles(name, layouts):
    """Tolerance: a sum of K fp32 products differs from the checker's by at most about K * 2^-24 of its largest partial sum
    (K <= 324 here: 2e-5 in the worst case, its square root typically), so 1e-5 of the layer's maximum as for the other fp32 cases."""
    case = conv_case(700, **FP32_TILES[name])
    plan, got, _ = run_conv(case, dn.MODE_FP32, layouts[0], layouts[1])
    assert plan.kernel == "direct_fp32"
    parity(got, oracle_conv(case), 1e-5)


FP32_SPLIT = {   # three bf16 parts: tiles of 32, 64 and 128 filters, ragged maps, K of one step and of a part of one, odd filters
    "32_filters_15_channels": dict(b=2, c=15, h=9, w=13, n=18, size=3),
    "64_filters_stride2_odd_map": dict(b=3, c=40, h=21, w=17, n=50, size=3, stride=2, act="logistic"),
    "128_filters_and_one": dict(b=1, c=33, h=11, w=19, n=129, size=3, act="linear"),
    "1x1_two_tiles_and_a_bit": dict(b=3, c=136, h=9, w=11, n=255, size=1),
    "1x1_one_pixel": dict(b=1, c=200, h=1, w=1, n=255, size=1),
    "5x5_no_padding": dict(b=2, c=8, h=12, w=9, n=33, size=5, pad=0),
    "several_tiles_an_sm": dict(b=4, c=16, h=150, w=141, n=40, size=3),
}


@pytest.mark.parametrize("name", list(FP32_SPLIT))
@pytest.mark.parametrize("layouts", [("nchw", "nchw"), ("nchw", "nhwc"), ("nhwc", "nhwc"), ("both", "nchw")])
def test_full_precision_on_the_tensor_cores(name, layouts, monkeypatch):
    """Each product is exact to about 2^-33 of its value and the sums of 32 channels are rounded as fp32 sums are; tolerance as for the
    CUDA-core kernel, and the root mean square of the error against 64-bit sums is no larger than that kernel's (a fifth is the
    spread of layers of a few hundred values)."""
    import numpy as np
    import torch
    case = conv_case(720, **dict(FP32_SPLIT[name], act="linear"))
    act = FP32_SPLIT[name].get("act", "leaky")
    t = {k: torch.from_numpy(np.asarray(case[k], np.float64)) for k in ("x", "w", "biases", "scales", "mean", "var")}
    exact = torch.nn.functional.conv2d(t["x"], t["w"], stride=case["stride"], padding=case["pad"])
    col = lambda v: v[:, None, None]  # noqa: E731
    exact = ((exact - col(t["mean"])) / (col(t["var"]).sqrt() + 1e-6) * col(t["scales"]) + col(t["biases"])).numpy()
    rms, layout = {}, "nchw" if layouts[0] == "both" else layouts[0]
    for knob in ("0", "1"):
        monkeypatch.setenv("DNB_FP32_TC", knob)
        plan, got, second = run_conv(case, dn.MODE_FP32, layout, layouts[1], both=layouts[0] == "both")
        assert plan.kernel == "direct_fp32" and ("three_bf16_parts" in plan.describe()) == (knob == "1"), plan.describe()
        assert second is None or np.array_equal(got, second)
        parity(got, exact, 1e-5)
        rms[knob] = np.sqrt(((got - exact) ** 2).mean())
    assert rms["1"] <= 1.2 * rms["0"], rms
    case["act"] = act
    _, got, _ = run_conv(case, dn.MODE_FP32, layout, layouts[1])
    parity(got, oracle_conv(case), 1e-5)


SPARSE = {   # what an output is made of: a product or a few of them among zeros, values of one sign
    "identity_1x1": dict(b=1, c=128, h=33, w=37, n=128, size=1),
    "few_inputs": dict(b=2, c=256, h=24, w=25, n=96, size=1),
    "few_inputs_3x3": dict(b=2, c=40, h=24, w=25, n=64, size=3),
    "few_weights_3x3": dict(b=2, c=64, h=24, w=25, n=130, size=3),
    "positive": dict(b=2, c=64, h=24, w=25, n=64, size=3, dist="uniform"),
    "wide_range": dict(b=2, c=128, h=24, w=25, n=64, size=1),
}


@pytest.mark.parametrize("name", list(SPARSE))
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
def test_full_precision_of_sparse_sums(name, layout, monkeypatch):
    """Sums of one or a few products are no further from 64 bits than the CUDA cores' (2 % and a tenth: the spread of the root mean square and of the largest error over some
    1e5 outputs), and a factor of 1 gives the input back to the bit."""
    import numpy as np
    import torch
    case = conv_case(723, **dict(SPARSE[name], act="linear", bn=False))
    case["biases"][...] = 0
    g = np.random.default_rng(724)
    x, w = case["x"], case["w"]
    K = w.shape[1] * w.shape[2] * w.shape[3]
    if name.startswith("identity"):
        w[:, :, 0, 0] = np.eye(128, dtype=np.float32)
        x *= np.exp2(g.integers(-30, 30, x.shape)).astype(np.float32)
    elif name.startswith("few_inputs"):
        x *= g.random(x.shape) < 2.5 / K
    elif name.startswith("few_weights"):
        w *= g.random(w.shape) < 2.5 / K
    elif name == "positive":
        w[...] = np.abs(w)
    else:
        x *= np.exp2(g.integers(-12, 12, x.shape)).astype(np.float32)
    exact = torch.nn.functional.conv2d(torch.from_numpy(x).double(), torch.from_numpy(w).double(), padding=case["pad"]).numpy()
    err = {}
    for knob in ("0", "1"):
        monkeypatch.setenv("DNB_FP32_TC", knob)
        plan, got, _ = run_conv(case, dn.MODE_FP32, layout, layout)
        assert (plan.describe() != "direct_fp32") == (knob == "1")
        d = np.abs(got - exact)
        some = exact != 0
        assert not got[~some].any()
        rel = d[some] / np.abs(exact[some])
        err[knob] = (float(np.sqrt((d ** 2).mean() / (exact ** 2).mean())), float(d.max() / np.abs(exact).max())) + ((float(np.sqrt((rel ** 2).mean())), float(rel.max())) if "few" in name else ())
        if name.startswith("identity"):
            assert np.array_equal(got, x), knob
    assert err["1"][0] <= 1.02 * err["0"][0] and err["1"][1] <= 1.1 * err["0"][1], err
    if "few" in name:   # of each output by itself, but for those that cancel
        assert err["1"][2] <= 1.5 * err["0"][2] or err["1"][3] <= 1.1 * err["0"][3], err


def test_full_precision_on_the_tensor_cores_out_of_range(monkeypatch):
    """Infinities, NaN, values whose high half or whose sum overflows, and sums too small for low halves: bit for bit what the
    CUDA-core kernel makes of them where that is not finite or tiny, close to it elsewhere."""
    import numpy as np
    case = conv_case(721, b=2, c=16, h=14, w=15, n=40, size=3, act="linear", bn=False)
    case["biases"][...] = 0
    x = case["x"]
    x[0, 3, 4, 5], x[0, 0, 10, 2], x[1, 7, 0, 0], x[1, 2, 8, 8] = np.inf, np.nan, -np.inf, np.float32(3.4028235e38)
    case["w"][5, :, 1, 1] = 0                                     # infinity times zero
    x[1, :, 10:14, 10:15] *= np.float32(1e-33)
    out = {}
    for layout in ("nchw", "nhwc"):
        for knob in ("0", "1"):
            monkeypatch.setenv("DNB_FP32_TC", knob)
            plan, out[knob], _ = run_conv(case, dn.MODE_FP32, "nchw", layout)
            assert ("three_bf16_parts" in plan.describe()) == (knob == "1")
        odd = ~np.isfinite(out["0"])
        tiny = np.abs(out["0"]) < 2.0 ** -91
        assert odd.any() and tiny.any() and np.array_equal(np.isfinite(out["1"]), ~odd)
        assert np.array_equal(out["0"][odd], out["1"][odd], equal_nan=True) and np.array_equal(out["0"][tiny], out["1"][tiny])
        plain = ~odd & ~tiny & (np.abs(out["0"]) < 1e30)
        assert np.abs(out["0"][plain] - out["1"][plain]).max() <= 1e-5 * np.abs(out["0"][plain]).max()


@pytest.mark.parametrize("name,x_exp,w_exp", [("tiny_inputs_huge_weights", -118, 40), ("products_below_normal_numbers", -70, -40), ("at_the_line", -52, -38), ("tiny_weights", 30, -60), ("subnormal_weights", 100, -140)])
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
def test_full_precision_of_tiny_operands(name, x_exp, w_exp, layout, monkeypatch):
    """Rows of pixels whose operands' parts or products are not normal numbers beside rows of ordinary size: tiny ones as the CUDA-core kernel adds
    them, to the bit; layers with tiny weights run there altogether."""
    import numpy as np
    case = conv_case(729, b=2, c=80, h=21, w=23, n=72, size=3, act="linear", bn=False)
    case["biases"][...] = 0
    x, w = case["x"], case["w"]
    w[...] = np.sign(w) * np.exp2(w_exp + np.abs(w) * 4).astype(np.float32)
    x[:, :, 6:13] = (x[:, :, 6:13].astype(np.float64) * 2.0 ** x_exp).astype(np.float32)
    x[1, :, 16] = 0
    out = {}
    for knob in ("0", "1"):
        monkeypatch.setenv("DNB_FP32_TC", knob)
        plan, out[knob], _ = run_conv(case, dn.MODE_FP32, layout, layout)
        assert ("three_bf16_parts" in plan.describe()) == (knob == "1" and w_exp >= -45)
    assert np.isfinite(out["0"]).all() and out["0"][:, :, 8:11].any()
    if layout == "nchw" and name != "at_the_line":     # over channels-last tensors the CUDA-core kernel's order is another
        assert np.array_equal(out["0"][:, :, 7:12], out["1"][:, :, 7:12])
    for rows in (slice(0, 5), slice(8, 11), slice(14, None)):
        scale = np.abs(out["0"][:, :, rows]).max()
        assert np.abs(out["1"][:, :, rows] - out["0"][:, :, rows].astype(np.float64)).max() <= 2e-6 * scale


@pytest.mark.parametrize("shape", [dict(b=4, c=64, h=52, w=51, n=200, size=3), dict(b=2, c=15, h=33, w=40, n=30, size=3, stride=2), dict(b=3, c=131, h=26, w=27, n=64, size=1)])
@pytest.mark.parametrize("layouts", [("nchw", "nchw"), ("nchw", "nhwc"), ("nhwc", "nhwc")])
def test_full_precision_without_finite_sums(shape, layouts, monkeypatch):
    """Every sum infinite or NaN, and one pixel in a hundred: what the CUDA cores make of it, in a few times their time (not in 60 and more)."""
    import numpy as np
    import torch
    from gpu_util import dev_nchw, dev_nhwc, empty_nchw, empty_nhwc
    case = conv_case(727, **dict(shape, act="linear", bn=False))
    g = np.random.default_rng(728)
    b, c, h, w = case["x"].shape
    n, size = case["w"].shape[0], case["w"].shape[2]
    few = case["x"].copy()
    few[g.random(few.shape) < 0.01 / c] = np.inf
    every = np.full_like(few, np.nan)
    every[:, :, ::2] = -np.inf
    for x in (few, every):
        out, us = {}, {}
        for knob in ("0", "1"):
            monkeypatch.setenv("DNB_FP32_TC", knob)
            plan = dn.ConvPlan(b, c, h, w, n, size, case["stride"], case["pad"], 1, False, "linear", False, dn.MODE_FP32)
            plan.set_params(case["w"], case["biases"])
            xt, xd = dev_nchw(x) if layouts[0] == "nchw" else dev_nhwc(x)
            yt, yd = (empty_nchw if layouts[1] == "nchw" else empty_nhwc)(b, n, plan.out_h, plan.out_w)
            times = []
            for _ in range(3):
                e0, e1 = torch.cuda.Event(True), torch.cuda.Event(True)
                e0.record()
                plan.forward(xd, yd)
                e1.record()
                torch.cuda.synchronize()
                times.append(e0.elapsed_time(e1) * 1e3)
            plan.check_status()
            us[knob] = min(times)
            out[knob] = yt.cpu().numpy()
        odd = ~np.isfinite(out["0"])
        assert odd.any() and np.array_equal(np.isfinite(out["1"]), ~odd) and np.array_equal(out["0"][odd], out["1"][odd], equal_nan=True)
        if not odd.all():
            parity(out["1"][~odd], out["0"][~odd], 1e-5)
        assert us["1"] < 8 * us["0"] + 50, us


@pytest.mark.parametrize("shape", [dict(b=4, c=64, h=52, w=51, n=128, size=3), dict(b=2, c=40, h=61, w=64, n=60, size=3, stride=2), dict(b=4, c=128, h=52, w=52, n=64, size=1)])
def test_full_precision_plan_in_several_hands(shape, monkeypatch):
    """One FP32 plan over different Darknet tensors on two streams at once, from two threads at once, and captured before its first plain
    call: every output is the one of a call by itself, to the bit, and no call takes device memory."""
    import threading

    import numpy as np
    import torch
    monkeypatch.setenv("DNB_FP32_TC", "1")
    case = conv_case(725, **shape)
    b, c, h, w = case["x"].shape
    n, size = case["w"].shape[0], case["w"].shape[2]
    plan = dn.ConvPlan(b, c, h, w, n, size, case["stride"], case["pad"], 1, True, "leaky", False, dn.MODE_FP32)
    plan.set_params(case["w"], case["biases"], case["scales"], case["mean"], case["var"])
    xs = [torch.from_numpy(case["x"] * np.float32(f)).cuda() for f in (1, -2, 3, 0.5)]
    ys = [torch.empty(b, n, plan.out_h, plan.out_w, device="cuda") for _ in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    forward = lambda i, out: plan.forward(dn.as_tensor(xs[i], dn.NCHW), dn.as_tensor(out, dn.NCHW), stream=streams[i].cuda_stream)  # noqa: E731
    torch.cuda.synchronize()
    warm = dn.ConvPlan(b, c, h, w, n, size, case["stride"], case["pad"], 1, True, "leaky", False, dn.MODE_FP32)   # loads the kernel
    warm.set_params(case["w"], case["biases"], case["scales"], case["mean"], case["var"])
    warm.forward(dn.as_tensor(xs[0], dn.NCHW), dn.as_tensor(ys[0], dn.NCHW))
    torch.cuda.synchronize()
    taken = lambda: -torch.cuda.mem_get_info()[0] - torch.cuda.memory_reserved()  # noqa: E731
    before = taken()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[0]):
        forward(0, ys[0])
    graph.replay()
    torch.cuda.synchronize()
    captured = ys[0].clone()
    want = []
    for i in range(len(xs)):
        forward(i, ys[i])
        torch.cuda.synchronize()
        want.append(ys[i].clone())
    assert torch.equal(captured, want[0])
    parity(want[0].cpu().numpy(), oracle_conv(case), 1e-5)
    for _ in range(3):
        for y in ys:
            y.zero_()
        torch.cuda.synchronize()
        for _ in range(8):                                     # calls of two and more streams in flight together
            for i in range(len(xs)):
                forward(i, ys[i])
        torch.cuda.synchronize()
        assert all(torch.equal(y, v) for y, v in zip(ys, want))
    for y in ys:
        y.zero_()
    torch.cuda.synchronize()
    threads = [threading.Thread(target=lambda i=i: [forward(i, ys[i]) for _ in range(50)]) for i in range(len(xs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    plan.check_status()
    assert all(torch.equal(y, v) for y, v in zip(ys, want))
    assert taken() - before < 8 << 20                          # the graph's own; a copy of one input would be 2.6 MB for each stream and call
    graph.reset()


def test_full_precision_wait_expiry(monkeypatch):
    """A withheld operand load: the bounded wait runs out, the call reports it, and the next launch is right."""
    import torch
    monkeypatch.setenv("DNB_FP32_TC", "1")
    case = conv_case(722, b=2, c=48, h=20, w=20, n=100, size=3)
    plan = dn.ConvPlan(2, 48, 20, 20, 100, 3, 1, 1, 1, True, "leaky", False, dn.MODE_FP32)
    plan.set_params(case["w"], case["biases"], case["scales"], case["mean"], case["var"])
    x = torch.from_numpy(case["x"]).cuda()
    y = torch.empty(2, 100, 20, 20, device="cuda")
    plan.set_diagnostics(4_000_000, 32)
    plan.forward(dn.as_tensor(x, dn.NCHW), dn.as_tensor(y, dn.NCHW))
    with pytest.raises(dn.DarknetB200Error) as e:
        plan.check_status()
    assert e.value.status == dn.ETIMEOUT
    plan.set_diagnostics(0, 0)
    plan.forward(dn.as_tensor(x, dn.NCHW), dn.as_tensor(y, dn.NCHW))
    plan.check_status()
    parity(y.cpu().numpy(), oracle_conv(case), 1e-5)


@pytest.mark.parametrize("mode", [dn.MODE_TF32, dn.MODE_FP32])
def test_first_call_from_a_new_host_thread(mode, monkeypatch):
    """A thread that has not used the GPU yet runs a plan for tensors that it has not run for: equal to the same call from here."""
    import threading

    import torch
    from gpu_util import dev_nhwc
    monkeypatch.setenv("DNB_FP32_TC", "1")
    case = conv_case(726, b=1, c=64, h=19, w=19, n=64, size=3)
    plan = dn.ConvPlan(1, 64, 19, 19, 64, 3, 1, 1, 1, True, "leaky", False, mode)
    plan.set_params(case["w"], case["biases"], case["scales"], case["mean"], case["var"])
    xt, xd = dev_nhwc(case["x"])
    ys = [torch.zeros(1, 64, 19, 19, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    stream = torch.cuda.current_stream().cuda_stream
    yd = [dn.as_tensor(y, dn.NCHW) for y in ys]
    failed = []

    def other():
        try:
            plan.forward(xd, yd[0], stream=stream)
        except dn.DarknetB200Error as e:
            failed.append(e)

    t = threading.Thread(target=other)
    t.start()
    t.join()
    assert not failed, failed
    plan.forward(xd, yd[1], stream=stream)
    torch.cuda.synchronize()
    assert torch.equal(*ys)
    parity(ys[0].cpu().numpy(), oracle_conv(case), 1e-2 if mode == dn.MODE_TF32 else 1e-5)


@pytest.mark.parametrize("name", ["groups_of_four_channels", "groups_off_four_channel_boundary", "slab_4"])
def test_grouped_layers_with_bf16_storage(name):
    """A grouped layer of a BF16 network: bf16 in, fp32 sums, bf16 out.  The input is rounded first, so what is left is the
    output's rounding, 2^-9 of each value."""
    from gpu_util import bf16_round
    case = conv_case(701, **FP32_TILES[name])
    case["x"] = bf16_round(case["x"])
    _, got, _ = run_conv(case, dn.MODE_BF16, "nhwc", "nhwc")
    parity(got, oracle_conv(case), 2 ** -8)


SPLIT_TILES = {   # (case, K ranges): one tile per cluster, the K loop cut across it
    "ranges_longer_than_the_ring": (dict(b=1, c=512, h=9, w=13, n=40, size=3), "2"),
    "uneven_ranges": (dict(b=1, c=48, h=11, w=7, n=33, size=3), "5"),
    "fewer_rows_than_ranges": (dict(b=1, c=1024, h=1, w=5, n=100, size=1), "8"),
    "one_filter_over_a_tile": (dict(b=2, c=64, h=10, w=12, n=257, size=3, act="linear"), "3"),
    "flat_batch_ragged": (dict(b=3, c=256, h=7, w=11, n=72, size=1, act="logistic"), "4"),
    "stride2_odd_map": (dict(b=2, c=40, h=21, w=17, n=24, size=3, stride=2), "6"),
    "narrow_rows": (dict(b=2, c=16, h=12, w=10, n=20, size=3), "2"),
    "pairs_odd_pixel_tiles": (dict(b=1, c=128, h=17, w=19, n=512, size=3), "7"),
}


@pytest.mark.parametrize("name", list(SPLIT_TILES))
@pytest.mark.parametrize("mode,tol", [(dn.MODE_TF32, 1e-2), (dn.MODE_BF16, 3e-2)])
def test_one_tile_per_cluster(name, mode, tol, monkeypatch):
    """Tolerances are the tensor-core kernel's (the products' 10 or 7 mantissa bits); the two layouts of one launch are bit-equal."""
    shape, ranges = SPLIT_TILES[name]
    monkeypatch.setenv("DNB_TC_SPLITK", ranges)
    case = conv_case(710, **shape)
    want = oracle_conv(case)
    plan, got, _ = run_conv(case, mode, "nhwc", "nhwc")
    assert f"splits={ranges}" in plan.describe() and "one_tile_per_cluster" in plan.describe(), plan.describe()
    parity(got, want, tol)
    _, nchw, nhwc = run_conv(case, mode, "nchw", "nchw", both=True)
    assert (nchw == nhwc).all()
    parity(nchw, want, tol)
    _, alone, _ = run_conv(case, mode, "nchw", "nchw")
    parity(alone, want, tol)


@pytest.mark.parametrize("shape", [dict(b=1, c=96, h=9, w=7, n=64, size=3), dict(b=2, c=256, h=7, w=7, n=40, size=1)])
@pytest.mark.parametrize("ranges", ["2", "6"])
def test_one_tile_per_cluster_integer_sums(shape, ranges, monkeypatch):
    """The int8 kind: the ranges' integer sums are exact, so they equal the uncut kernel's whatever the cut."""
    import numpy as np
    case = conv_case(711, **shape)
    monkeypatch.setenv("DNB_TC_SPLITK", "0")
    _, whole, _ = run_conv(case, dn.MODE_TF32, "nhwc", "nhwc", xnor=True)
    monkeypatch.setenv("DNB_TC_SPLITK", ranges)
    _, got, _ = run_conv(case, dn.MODE_TF32, "nhwc", "nhwc", xnor=True)
    assert np.array_equal(got, whole)


def test_predict_from_ordinary_and_page_locked_memory(tmp_path):
    """The same images from ordinary host memory (carried over chunk by chunk), at an odd address, and from page-locked memory:
    sizes below one chunk, a few chunks, and more chunks than the staging ring has slots; first, captured and replayed steps."""
    import numpy as np
    import torch
    from darknet_b200 import synth
    for batch, size in ((1, 32), (1, 450), (24, 512)):
        cfg = (synth._net(batch, size, size) + synth._conv(16, 3, stride=2) + "\n[avgpool]\n" + synth._conv(10, 1, bn=False, act="linear"))
        path = str(tmp_path / "n.weights")
        synth.write_weights(path, synth.seeded_params(cfg, 1))
        net = dn.Network(cfg, path, dn.MODE_TF32, text=True)
        x = [synth.seeded_input(cfg, k) for k in range(2)]
        want = [net.predict(torch.from_numpy(a).pin_memory()).copy() for a in x]
        assert not np.array_equal(want[0], want[1])
        odd = np.empty(x[0].size + 1, np.float32)[1:]
        for k in (0, 1, 1, 0, 0):
            odd[:] = x[k].reshape(-1)
            assert np.array_equal(net.predict(x[k]), want[k])
            assert np.array_equal(net.predict(odd), want[k])
        net.submit(x[1])
        net.submit(x[0])
        assert np.array_equal(net.collect(), want[1]) and np.array_equal(net.collect(), want[0])
        net.close()


@pytest.mark.parametrize("batch,size,what", [(1, 16, "one_tile_per_cluster"), (3, 18, ""), (40, 44, "pair=1")])
@pytest.mark.parametrize("mode,tol", [(dn.MODE_TF32, 1e-2), (dn.MODE_BF16, 3e-2)])
def test_shortcut_of_another_shape_in_the_epilogue(batch, size, what, mode, tol, tmp_path):
    """ResNet's stage boundaries in one launch each: the addend has fewer channels, and twice the map (every second pixel counts).
    Against the checker layer by layer (four convolutions deep: the kernel tests' tolerances still hold)."""
    from darknet_b200 import synth
    from oracle import network as orc
    cfg = (synth._net(batch, size, size, 16) + synth._conv(64, 3) + synth._conv(512, 3, stride=2, act="linear") + synth._shortcut(-2, "leaky") +
           synth._conv(64, 1) + synth._conv(192, 1, act="linear") + synth._shortcut(-2, "leaky"))
    params = synth.seeded_params(cfg, 5)
    path = str(tmp_path / "s.weights")
    synth.write_weights(path, params)
    x = synth.seeded_input(cfg, 6, "normal")
    want = orc.forward_network(cfg, params, x)
    net = dn.Network(cfg, path, mode, text=True)
    net.predict(x)
    assert what in net.layer_describe(1), net.layer_describe(1)
    for i in (2, 5):
        parity(net.layer_output(i), want[i], tol, f"layer {i}")
    for i in (1, 4):                     # made from the convolution's input on request: a step does not write it
        parity(net.layer_output(i), want[i], tol, f"layer {i}")
        assert (net.layer_output_images(i, batch - 1) == net.layer_output(i)[batch - 1:]).all()
    for i in (2, 5):                     # ... and what the step wrote is still there, as is what the next one writes
        parity(net.layer_output(i), want[i], tol, f"layer {i}")
    again = net.predict(x).copy()
    assert (net.predict(x) == again).all()
    parity(net.layer_output(5), want[5], tol, "layer 5")


@pytest.mark.parametrize("name,shape", [
    ("5x5_s2_one_row_over", dict(b=2, c=3, h=34, w=35, n=48, size=5, stride=2)),
    ("3x3_s2_gray_narrower_than_a_tile", dict(b=3, c=1, h=3, w=9, n=16, size=3, stride=2)),
    ("7x7_one_pixel", dict(b=2, c=3, h=1, w=1, n=16, size=7, act="logistic")),
    ("3x3_two_channels_one_column_over", dict(b=1, c=2, h=33, w=17, n=32, size=3)),
])
@pytest.mark.parametrize("mode,tol", [(dn.MODE_TF32, 1e-2), (dn.MODE_BF16, 3e-2)])
def test_first_layer_patches(name, shape, mode, tol):
    """8 x 16 pixel tiles whose rows are read from the image's patch.  Tolerance as for the other first-layer cases: operands rounded
    to TF32 (2^-11), K <= 147 of them, and for BF16 networks an output rounded to 2^-9."""
    case = conv_case(710, **shape)
    plan, got, _ = run_conv(case, mode, "nchw", "nhwc")
    assert plan.kernel == "stem_tc_tf32"
    parity(got, oracle_conv(case), tol, name)


@pytest.mark.parametrize("size,filters", [(256, 32), (255, 8)])   # 255 x 255 x 8 in bf16: only whole eighths are 128-byte multiples
@pytest.mark.parametrize("mode", [dn.MODE_TF32, dn.MODE_BF16])
def test_steps_in_parts(size, filters, mode, tmp_path):
    """A step whose upload and last pull are worth cutting up: first layers by parts, last ones by halves, a [yolo] layer, a
    [route] and a fused and an unfused [shortcut] inside them.  A pixel's sums run in one order whatever the batch, so the step's results are the
    whole-batch pass's to the bit: first, captured and replayed steps, one alone and two in flight."""
    import numpy as np
    import torch
    from darknet_b200 import synth
    yolo = synth._yolo("0,1", "10,14, 23,27", 2, 40)
    cfg = (synth._net(16, size, size) + synth._conv(filters, 3) + synth._conv(64, 3, stride=2) + synth._conv(64, 1) + synth._conv(64, 3) +
           synth._shortcut(-3) + synth._conv(512, 3, stride=2) + synth._conv(90, 1, bn=False, act="linear") + yolo + "\n[route]\nlayers=-4\n" +
           synth._conv(512, 3) + synth._conv(512, 3) + synth._conv(64, 1) + synth._shortcut(-4) + synth._conv(512, 3) + synth._conv(90, 1, bn=False, act="linear") + yolo)
    path = str(tmp_path / "p.weights")
    synth.write_weights(path, synth.seeded_params(cfg, 3))
    net = dn.Network(cfg, path, mode, text=True)
    heads = [i for i in range(net.n) if net.layer_type(i) == "yolo"]
    x = [synth.seeded_input(cfg, k) for k in range(2)]
    want = []
    for a in x:
        net.forward(torch.from_numpy(a).cuda())
        torch.cuda.synchronize()
        want.append([net.layer_output(i) for i in [4] + heads])
    assert len(heads) == 2 and not np.array_equal(want[0][2], want[1][2])
    pinned = [torch.from_numpy(a).pin_memory() for a in x]
    for k in (0, 1, 0, 1, 1):
        for images in (x[k], pinned[k]):
            assert np.array_equal(net.predict(images).reshape(-1), want[k][2].reshape(-1))
            assert np.array_equal(net.yolo_output(heads[0]).reshape(-1), want[k][1].reshape(-1))
            assert np.array_equal(net.layer_output(4), want[k][0])
    for _ in range(2):
        net.submit(pinned[1])
        net.submit(x[0])
        for k in (1, 0):
            assert np.array_equal(net.collect().reshape(-1), want[k][2].reshape(-1))
            assert np.array_equal(net.yolo_output(heads[0]).reshape(-1), want[k][1].reshape(-1))
    net.close()


@pytest.mark.parametrize("c,h,w,pitch", [(33, 3, 43, 40), (32, 8, 16, 32), (5, 11, 3, 8), (70, 1, 257, 72), (64, 4, 8, 64)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_to_channels_last_tiles(c, h, w, pitch, dtype):
    """Darknet's layout to channels-last in tiles of 32 channels x 128 pixels: one pixel or channel over a tile, padding channels
    (zeroed).  A copy: the values are the input's, rounded to bf16 where that is the storage type."""
    import torch
    x = torch.randn(2, c, h, w, generator=torch.Generator().manual_seed(1)).cuda()
    y = torch.full((2, h, w, pitch), 7.0, dtype=getattr(torch, dtype), device="cuda")
    dn.convert(dn.as_tensor(x, dn.NCHW), dn.as_tensor(y, dn.NHWC, c))
    torch.cuda.synchronize()
    assert torch.equal(y[..., :c], x.permute(0, 2, 3, 1).to(y.dtype)) and not y[..., c:].any()


def test_first_layer_of_a_very_long_image():
    """A row of 2^25 + 37 pixels: beyond the offsets of the patch kernel.  Windows of the row against the checker (whose image is the
    window and a pixel on each side); operands rounded to TF32."""
    import numpy as np
    import torch
    from conftest import rel_to_max
    w = (1 << 25) + 37
    plan = dn.ConvPlan(1, 3, 1, w, 16, 3, 1, 1, 1, False, "linear")
    g = np.random.Generator(np.random.Philox(key=[9, 9]))
    wt, bias = g.standard_normal((16, 3, 3, 3), dtype=np.float32), g.standard_normal(16, dtype=np.float32)
    plan.set_params(wt, bias)
    x = torch.randn(1, 3, 1, w, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda")
    y = torch.full((1, 1, w, 16), float("nan"), device="cuda")
    plan.forward(dn.as_tensor(x, dn.NCHW), dn.as_tensor(y, dn.NHWC, 16))
    plan.check_status()
    from oracle import network as orc
    for at in (0, 1000, (1 << 24) - 8, (1 << 25) - 20, w - 300):
        lo, hi = max(at - 1, 0), min(at + 301, w)
        want = orc.conv_forward(x[..., lo:hi].cpu().numpy(), wt, bias, None, None, None, stride=1, pad=1, groups=1, activation="linear")
        want = want[..., at - lo:at - lo + 300]
        got = y[:, :, at:at + 300].permute(0, 3, 1, 2).cpu().numpy()
        assert rel_to_max(got, want) < 1e-2
    del x, y
    torch.cuda.empty_cache()


@pytest.mark.parametrize("mode,c,pair", [(dn.MODE_BF16, 64, 0), (dn.MODE_BF16, 72, 1), (dn.MODE_TF32, 32, 0), (dn.MODE_TF32, 40, 1)])
def test_pairs_start_at_sixteen_iterations(mode, c, pair, monkeypatch):
    """3x3 over one block of channels (nine iterations) runs as single CTAs, over two as pairs."""
    monkeypatch.delenv("DNB_TC_PAIR", raising=False)
    case = conv_case(712, b=8, c=c, h=38, w=38, n=512, size=3)
    plan, got, _ = run_conv(case, mode, "nhwc", "nhwc")
    assert f"pair={pair}" in plan.describe() and "splits=1" in plan.describe(), plan.describe()
    parity(got, oracle_conv(case), 3e-2 if mode == dn.MODE_BF16 else 1e-2)


TWO_GROUPS = {   # (case, in / out layout, residual, xnor): launches whose CTAs have two groups of epilogue warps, at odd sizes
    "pair_residual_odd_tiles": (dict(b=61, c=64, h=19, w=17, n=256, size=3), "nhwc", True, False),
    "pair_residual_two_filter_tiles": (dict(b=73, c=1024, h=11, w=13, n=512, size=1), "nhwc", True, False),
    "pair_short_loop": (dict(b=73, c=72, h=13, w=21, n=256, size=3), "nhwc", False, False),
    "darknet_layout_half_a_chunk_over": (dict(b=40, c=256, h=13, w=19, n=272, size=3), "nchw", False, False),
    "darknet_layout_fewer_filters_than_a_chunk": (dict(b=3, c=64, h=33, w=21, n=24, size=3), "nchw", False, False),
    "xnor_one_chunk": (dict(b=5, c=96, h=11, w=13, n=32, size=3), "nhwc", False, True),
    "xnor_ragged": (dict(b=70, c=256, h=14, w=15, n=200, size=1), "nhwc", False, True),
}


@pytest.mark.parametrize("name", list(TWO_GROUPS))
@pytest.mark.parametrize("mode", [dn.MODE_TF32, dn.MODE_BF16])
def test_two_epilogue_groups(name, mode, monkeypatch):
    """The second group of epilogue warps changes who finishes a value, not how: equal to one group's output to the bit (pairs with a residual,
    which always have two: to the convolution's own output plus the residual, rounded once more)."""
    import ctypes as C
    import numpy as np
    import torch
    from gpu_util import dev_nhwc, empty_nhwc, host_from_nhwc
    shape, layout, residual, xnor = TWO_GROUPS[name]
    if xnor and mode == dn.MODE_BF16:
        pytest.skip("xnor layers have one kind")
    case = conv_case(730, **shape)
    monkeypatch.setenv("DNB_TC_SPLITK", "0")
    out = {}
    for groups in ("1", "2"):
        monkeypatch.setenv("DNB_TC_EPI", groups)
        plan, out[groups], _ = run_conv(case, mode, "nhwc", layout, xnor=xnor)
        if not residual:
            assert f"epi={groups}" in plan.describe(), plan.describe()
    assert np.array_equal(out["1"], out["2"])
    if not residual:
        return
    store = torch.bfloat16 if mode == dn.MODE_BF16 else torch.float32
    add = np.random.Generator(np.random.Philox(key=[7, 7])).standard_normal(out["1"].shape, dtype=np.float32)
    xt, xd = dev_nhwc(case["x"], store)
    at, ad = dev_nhwc(add, store)
    yt, yd = empty_nhwc(*out["1"].shape, store)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    dn.check(dn.lib().dnb_conv_shortcut_forward(plan.handle, C.byref(xd), C.byref(ad), C.byref(yd), 1.0, 1.0, dn.ACTIVATIONS["linear"], stream))
    torch.cuda.synchronize()
    plan.check_status()
    assert "pair=1" in plan.describe() and "epi=2" in plan.describe(), plan.describe()
    parity(host_from_nhwc(yt, case["w"].shape[0]), out["1"] + host_from_nhwc(at, add.shape[1]), 2 ** -7 if mode == dn.MODE_BF16 else 2 ** -10)


@pytest.mark.parametrize("mode,xnor,batch,size", [
    (dn.MODE_TF32, False, 3, 60), (dn.MODE_TF32, False, 64, 22), (dn.MODE_BF16, False, 5, 68), (dn.MODE_TF32, True, 4, 60), (dn.MODE_TF32, True, 40, 28)])
@pytest.mark.parametrize("first_filters", [16, 32])
def test_maxpool_in_the_convolutions_epilogue(mode, xnor, batch, size, first_filters, tmp_path, monkeypatch):
    """Convolutions with the 2x2 maxpool after them in one launch against two launches, to the bit: maps that end inside a tile, filters
    beyond a staged chunk, signs for an xnor layer, filters whose every value is an infinity or NaN, the convolutions' own outputs."""
    import numpy as np
    from darknet_b200 import synth
    pool = "\n[maxpool]\nsize=2\nstride=2\n"
    cfg = (synth._net(batch, 4 * size, 4 * size) + synth._conv(first_filters, 3) + pool + synth._conv(72, 3, xnor=xnor) + pool + synth._conv(96, 3, xnor=xnor) + pool +
           synth._conv(128, 1, xnor=xnor) + synth._conv(160, 3, xnor=xnor) + "\n[avgpool]\n")
    params = synth.seeded_params(cfg, 8)
    params[0].biases[3] = -np.inf
    for f, v in ((0, np.inf), (1, -np.inf), (2, np.nan)):
        params[1].biases[f] = v
    path = str(tmp_path / "m.weights")
    synth.write_weights(path, params)
    import torch
    x, y = synth.seeded_input(cfg, 9, "normal"), synth.seeded_input(cfg, 10, "normal")
    stream, dev = torch.cuda.Stream(), None
    out = []
    for fuse in ("0", "1"):
        monkeypatch.setenv("DNB_FUSE_POOL", fuse)
        net = dn.Network(cfg, path, mode, text=True)
        launches = net.launches
        net.predict(x)
        got = [net.layer_output(i) for i in (1, 3, 5, 0, 2, 4, 6, 7)] + [net.predict(x).copy(), net.layer_output_images(2, batch - 1)]
        for graph in (False, True, True, True):      # the device's images are overwritten before the first layer's own output is asked for
            net.enable_graph(graph)
            dev = torch.from_numpy(x).cuda() if not graph else dev
            dev.copy_(torch.from_numpy(x))
            stream.wait_stream(torch.cuda.current_stream())
            net.forward(dev, stream=stream.cuda_stream)
            stream.synchronize()
            dev.zero_()
            got += [net.layer_output(i) for i in (0, 2, 7)]
        net.submit(x), net.submit(y)
        net.collect(), net.collect()
        got += [net.layer_output(i) for i in (0, 1, 7)]
        out.append(got + [launches])
        net.close()
    assert out[1][-1] < out[0][-1]
    for a, b in zip(*[o[:-1] for o in out]):
        assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("batch,size", [(2, 160), (40, 48)])
def test_own_output_of_a_first_xnor_layer_with_its_maxpool(batch, size, tmp_path):
    """The first layer's own output after a forward over a caller's buffer that is overwritten since: made from those images, not from a
    predict's before it or from nothing.  Equal to that of a predict over the same images, to the bit."""
    import numpy as np
    import torch
    from darknet_b200 import synth
    pool = "\n[maxpool]\nsize=2\nstride=2\n"
    cfg = synth._net(batch, size, size) + synth._conv(64, 3, xnor=True) + pool + synth._conv(32, 3, xnor=True) + "\n[avgpool]\n"
    params = synth.seeded_params(cfg, 11)
    path = str(tmp_path / "x.weights")
    synth.write_weights(path, params)
    x, y = synth.seeded_input(cfg, 12, "normal"), synth.seeded_input(cfg, 13, "normal")
    net = dn.Network(cfg, path, dn.MODE_TF32, text=True)
    net.predict(x)
    want = [net.layer_output(i) for i in range(net.n)]
    net.predict(y), net.predict(y)      # both of the network's own image buffers
    dev = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    net.forward(dev)
    torch.cuda.synchronize()
    dev.zero_()
    torch.cuda.synchronize()
    for i in range(net.n):
        assert np.array_equal(net.layer_output(i), want[i]), i
    net.close()


HALO = {   # one box for the nine taps, weights in shared memory: row widths, strides, channel blocks, ragged maps
    "tf32_64_byte_rows": (dict(b=3, c=16, h=37, w=27, n=32, size=3), dn.MODE_TF32, False),
    "tf32_two_blocks": (dict(b=2, c=40, h=33, w=18, n=48, size=3, act="linear"), dn.MODE_TF32, False),
    "tf32_stride2": (dict(b=2, c=24, h=63, w=37, n=32, size=3, stride=2), dn.MODE_TF32, False),
    "bf16_64_byte_rows": (dict(b=3, c=32, h=35, w=29, n=64, size=3), dn.MODE_BF16, False),
    "bf16_stride2_even_map": (dict(b=2, c=32, h=64, w=48, n=64, size=3, stride=2), dn.MODE_BF16, False),
    "int8_32_byte_rows": (dict(b=3, c=32, h=36, w=28, n=64, size=3), dn.MODE_TF32, True),
    "int8_64_byte_rows_stride2": (dict(b=2, c=64, h=41, w=33, n=80, size=3, stride=2), dn.MODE_TF32, True),
}


@pytest.mark.parametrize("name", list(HALO))
def test_one_box_for_nine_taps(name, monkeypatch):
    """Equal to the ordinary rings to the bit: the same products in the same order, in either layout."""
    import numpy as np
    shape, mode, xnor = HALO[name]
    case = conv_case(740, **shape)
    monkeypatch.setenv("DNB_TC_SPLITK", "0")
    out = {}
    for knob in ("0", "2"):
        monkeypatch.setenv("DNB_TC_HALO", knob)
        plan, a, b = run_conv(case, mode, "nhwc", "nchw", xnor=xnor, both=True)
        assert ("halo=1" in plan.describe()) == (knob == "2"), plan.describe()
        _, c, _ = run_conv(case, mode, "nhwc", "nhwc", xnor=xnor)
        assert np.array_equal(a, b) and np.array_equal(a, c)
        out[knob] = a
    assert np.array_equal(out["0"], out["2"])


@pytest.mark.parametrize("mode,c", [(dn.MODE_TF32, 512), (dn.MODE_BF16, 1024)])
def test_pairs_over_128_filters(mode, c, monkeypatch):
    """A launch of three rounds of such pairs where pairs over 256 filters or single CTAs take two of twice the length, on a ragged map: equal to single CTAs to the bit."""
    import numpy as np
    case = conv_case(750, b=15, c=c, h=25, w=27, n=512, size=1)
    monkeypatch.setenv("DNB_TC_SPLITK", "0")
    monkeypatch.delenv("DNB_TC_PAIR", raising=False)
    plan, got, _ = run_conv(case, mode, "nhwc", "nhwc")
    assert "pair=1" in plan.describe() and "bn=128" in plan.describe(), plan.describe()
    monkeypatch.setenv("DNB_TC_PAIR", "0")
    plan, single, _ = run_conv(case, mode, "nhwc", "nhwc")
    assert "pair=0" in plan.describe() and np.array_equal(got, single)
    parity(got, oracle_conv(case), 3e-2 if mode == dn.MODE_BF16 else 1e-2)


TAPS = {   # one load of pixels for the nine taps: tiles across rows and images, maps smaller than a tile, filters beyond a tile or a chunk, ragged blocks of channels
    "one_tile": dict(b=1, c=64, h=13, w=13, n=64, size=3),
    "rows_of_one_pixel": dict(b=33, c=64, h=3, w=1, n=48, size=3),
    "odd_pixel_tiles_residual": dict(b=2, c=96, h=19, w=19, n=128, size=3, act="linear"),
    "several_images_a_tile": dict(b=9, c=128, h=7, w=5, n=256, size=3),
    "half_a_chunk_ragged_channels": dict(b=4, c=72, h=26, w=25, n=200, size=3),
    "three_filter_tiles": dict(b=7, c=160, h=9, w=14, n=264, size=3, act="linear"),
    "wide_rows": dict(b=1, c=64, h=21, w=150, n=40, size=3),
    "rounds_of_tiles_residual": dict(b=9, c=64, h=38, w=38, n=512, size=3),
}


@pytest.mark.parametrize("boxes", ["0", "1"])
@pytest.mark.parametrize("name", list(TAPS))
@pytest.mark.parametrize("mode,tol", [(dn.MODE_TF32, 1e-2), (dn.MODE_BF16, 3e-2)])
def test_one_load_for_nine_taps(name, mode, tol, boxes, monkeypatch):
    """Whole numbers, whose sums are exact in any order: equal to the kernel that loads tap by tap to the bit, in either layout.  Others: within the mode's
    tolerance against the oracle; with a residual to the kernel's output plus it, rounded once more."""
    import ctypes as C
    import numpy as np
    import torch
    from gpu_util import dev_nhwc, empty_nhwc, host_from_nhwc, padding_is_zero
    case = conv_case(760, **TAPS[name])
    monkeypatch.setenv("DNB_TC_TAPS_BOX", boxes)
    whole = dict(case, x=np.rint(2 * case["x"]), w=np.rint(case["w"] / np.abs(case["w"]).max() * 6), biases=np.rint(9 * case["biases"]), scales=None, mean=None, var=None)
    out = {}
    for knob in ("0", "2"):
        monkeypatch.setenv("DNB_TC_TAPS", knob)
        plan, a, b = run_conv(whole, mode, "nhwc", "nchw", both=True)
        assert ("one_load_for_nine_taps" in plan.describe()) == (knob == "2"), plan.describe()
        assert (" boxes" in plan.describe()) == (knob == "2" and boxes == "1")
        plan, c, _ = run_conv(whole, mode, "nhwc", "nhwc")
        assert np.array_equal(a, b) and np.array_equal(a, c)
        out[knob] = a
    assert np.array_equal(out["0"], out["2"])
    plan, out["2"], _ = run_conv(case, mode, "nhwc", "nhwc")
    parity(out["2"], oracle_conv(case), tol)
    if "residual" not in name:
        return
    store = torch.bfloat16 if mode == dn.MODE_BF16 else torch.float32
    add = np.random.Generator(np.random.Philox(key=[8, 8])).standard_normal(out["2"].shape, dtype=np.float32)
    act2 = "leaky" if case["act"] == "linear" else "linear"
    xt, xd = dev_nhwc(case["x"], store)
    at, ad = dev_nhwc(add, store)
    yt, yd = empty_nhwc(*out["2"].shape, store)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    dn.check(dn.lib().dnb_conv_shortcut_forward(plan.handle, C.byref(xd), C.byref(ad), C.byref(yd), 1.0, 1.0, dn.ACTIVATIONS[act2], stream))
    torch.cuda.synchronize()
    plan.check_status()
    assert "one_load_for_nine_taps" in plan.describe(), plan.describe()
    want = out["2"] + host_from_nhwc(at, add.shape[1])
    if act2 == "leaky":
        want = np.where(want > 0, want, np.float32(0.1) * want)
    # both terms are rounded to the storage type (half an ulp of 11 or 8 bits each, and once more the sum)
    parity(host_from_nhwc(yt, add.shape[1]), want, 2 ** -7 if mode == dn.MODE_BF16 else 2 ** -10)
    assert padding_is_zero(yt, add.shape[1])


def test_one_load_for_nine_taps_wait_expiry(monkeypatch):
    """A withheld load makes a wait run out: the launch ends early, says so, and the next one is sound."""
    import numpy as np
    monkeypatch.setenv("DNB_TC_TAPS", "2")
    case = conv_case(761, b=3, c=64, h=30, w=30, n=64, size=3)
    plan, good, _ = run_conv(case, dn.MODE_TF32, "nhwc", "nhwc")
    from gpu_util import dev_nhwc, empty_nhwc, host_from_nhwc
    import torch
    xt, xd = dev_nhwc(case["x"])
    yt, yd = empty_nhwc(*good.shape)
    plan.set_diagnostics(4_000_000, 32)
    plan.forward(xd, yd)
    torch.cuda.synchronize()
    with pytest.raises(dn.DarknetB200Error) as e:
        plan.check_status()
    assert e.value.status == dn.ETIMEOUT
    plan.set_diagnostics(0, 0)
    plan.forward(xd, yd)
    torch.cuda.synchronize()
    plan.check_status()
    assert np.array_equal(host_from_nhwc(yt, good.shape[1]), good)


ONES = {   # 1x1 layers on the same kernel: pixels beyond the last tile, ragged channels, filters in place and in a ring, half a chunk of filters
    "in_place": dict(b=3, c=64, h=19, w=17, n=64, size=1),
    "one_pixel": dict(b=1, c=72, h=1, w=1, n=24, size=1, act="linear"),
    "in_place_two_filter_tiles": dict(b=5, c=96, h=13, w=14, n=320, size=1),
    "a_ring": dict(b=2, c=1032, h=13, w=13, n=250, size=1),
    "rounds_of_tiles": dict(b=9, c=128, h=52, w=51, n=255, size=1, act="linear", bn=False),
}


@pytest.mark.parametrize("name", list(ONES))
@pytest.mark.parametrize("mode,tol", [(dn.MODE_TF32, 1e-2), (dn.MODE_BF16, 3e-2)])
def test_1x1_layers_with_their_filters_in_place(name, mode, tol, monkeypatch):
    """The same products in the same order as in the kernel with a ring: equal to the bit, in either layout; with a [yolo] layer's logistic too."""
    import ctypes as C
    import numpy as np
    import torch
    from gpu_util import dev_nhwc, empty_nchw
    case = conv_case(770, **ONES[name])
    monkeypatch.setenv("DNB_TC_SPLITK", "0")
    out = {}
    for knob in ("0", "2"):
        monkeypatch.setenv("DNB_TC_TAPS", knob)
        plan, a, b = run_conv(case, mode, "nhwc", "nchw", both=True)
        assert ("one_load_for_a_block" in plan.describe()) == (knob == "2"), plan.describe()
        _, c, _ = run_conv(case, mode, "nhwc", "nhwc")
        _, d, _ = run_conv(case, mode, "nchw", "nchw")
        assert np.array_equal(a, b) and np.array_equal(a, c)
        out[knob] = [a, d]
        if case["act"] == "linear":
            n = a.shape[1]
            xt, xd = dev_nhwc(case["x"], torch.bfloat16 if mode == dn.MODE_BF16 else torch.float32)
            yt, yd = empty_nchw(*a.shape)
            stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
            dn.check(dn.lib().dnb_conv_yolo_forward(plan.handle, C.byref(xd), C.byref(yd), 3, n // 3 - 5, stream))
            torch.cuda.synchronize()
            plan.check_status()
            out[knob].append(yt.cpu().numpy())
    for a, b in zip(out["0"], out["2"]):
        assert np.array_equal(a, b)
    parity(out["2"][0], oracle_conv(case), tol)


@pytest.mark.parametrize("filters", [128, 192, 250])     # tiles of 64: with 74 pairs of CTAs a pair meets one of two, all of three, two of four
@pytest.mark.parametrize("batch,height,width", [(1, 13, 13), (9, 52, 51)])     # one tile a pair; four rounds and more
@pytest.mark.parametrize("mode", [dn.MODE_TF32, dn.MODE_BF16])
def test_a_pair_loads_the_filters_that_it_multiplies(filters, batch, height, width, mode, monkeypatch):
    """1x1 layers with several filter tiles in place: equal to the kernel with a ring to the bit, in either layout."""
    import numpy as np
    case = conv_case(775, b=batch, c=72, h=height, w=width, n=filters, size=1)
    monkeypatch.setenv("DNB_TC_SPLITK", "0")
    monkeypatch.setenv("DNB_TC_TAPS_BN", "64")
    out = {}
    for knob in ("0", "2"):
        monkeypatch.setenv("DNB_TC_TAPS", knob)
        plan, a, b = run_conv(case, mode, "nhwc", "nchw", both=True)
        assert ("one_load_for_a_block resident" in plan.describe()) == (knob == "2"), plan.describe()
        assert knob == "0" or "bn=64" in plan.describe(), plan.describe()
        out[knob] = a
        assert np.array_equal(a, b)
    assert np.array_equal(out["0"], out["2"])


def test_filters_in_place_by_themselves(monkeypatch):
    """A layer that takes two filter tiles in place without a knob, of which a pair meets one: equal to the kernel with a ring to the bit."""
    import numpy as np
    for knob in ("DNB_TC_TAPS", "DNB_TC_SPLITK", "DNB_TC_PAIR"):
        monkeypatch.delenv(knob, raising=False)
    case = conv_case(777, b=32, c=256, h=38, w=38, n=512, size=1)
    plan, got, _ = run_conv(case, dn.MODE_BF16, "nhwc", "nhwc")
    assert "bn=256" in plan.describe() and "one_load_for_a_block resident" in plan.describe(), plan.describe()
    monkeypatch.setenv("DNB_TC_TAPS", "0")
    plan, want, _ = run_conv(case, dn.MODE_BF16, "nhwc", "nhwc")
    assert "one_load" not in plan.describe() and np.array_equal(got, want)


@pytest.mark.parametrize("filters", [16, 40, 80, 200, 232])
@pytest.mark.parametrize("size", [1, 3])
def test_pairs_multiply_columns_in_steps_of_32(filters, size, monkeypatch):
    """Layers whose filters are an odd number of sixteens: whole numbers, equal to single CTAs to the bit, in either layout."""
    import re
    import numpy as np
    case = conv_case(776, b=2, c=64, h=19, w=18, n=filters, size=size)
    case = dict(case, x=np.rint(2 * case["x"]), w=np.rint(case["w"] / np.abs(case["w"]).max() * 6), biases=np.rint(9 * case["biases"]), scales=None, mean=None, var=None)
    monkeypatch.setenv("DNB_TC_SPLITK", "0")
    out = {}
    for knob in ("0", "2"):
        monkeypatch.setenv("DNB_TC_TAPS", knob)
        plan, a, b = run_conv(case, dn.MODE_TF32, "nhwc", "nchw", both=True)
        assert ("one_load_for" in plan.describe()) == (knob == "2"), plan.describe()
        assert knob == "0" or int(re.search(r"bn=(\d+)", plan.describe()).group(1)) % 32 == 0, plan.describe()
        assert np.array_equal(a, b)
        out[knob] = a
    assert np.array_equal(out["0"], out["2"])


@pytest.mark.parametrize("mode,tail", [(dn.MODE_TF32, "yolo"), (dn.MODE_BF16, "yolo"), (dn.MODE_TF32, "softmax"), (dn.MODE_TF32, "xnor")])
def test_networks_that_keep_the_order_of_their_sums(mode, tail, tmp_path, monkeypatch):
    """3x3 layers over several blocks of channels, of a size that takes the kernel with one load for nine taps by itself, whose sums run in another order: a TF32
    detector's do; those of networks whose sums keep theirs (bf16, a [softmax], xnor layers), however few their layers, do not, and the outputs are what they are without that kernel, to the bit."""
    import numpy as np
    from darknet_b200 import synth
    layers = synth._conv(64, 3) + synth._conv(120, 3) + synth._conv(128, 3)
    if tail == "yolo":
        layers += synth._conv(90, 1, bn=False, act="linear") + synth._yolo("0,1", "10,14, 23,27", 2, 40)
    elif tail == "softmax":
        layers += synth._conv(90, 1, bn=False, act="linear") + "\n[avgpool]\n\n[softmax]\ngroups=1\n"
    else:
        layers += synth._conv(64, 3, xnor=True) + "\n[avgpool]\n"
    cfg = synth._net(12, 128, 128) + layers
    path = str(tmp_path / "o.weights")
    synth.write_weights(path, synth.seeded_params(cfg, 25))
    x = synth.seeded_input(cfg, 26)
    out = []
    for knob in (None, "0"):
        monkeypatch.delenv("DNB_TC_TAPS", raising=False)
        if knob:
            monkeypatch.setenv("DNB_TC_TAPS", knob)
        net = dn.Network(cfg, path, mode, text=True)
        result = net.predict(x).copy()
        out.append((net.layer_output(2), result))
        moved = "one_load_for_nine_taps" in net.layer_describe(2)
        assert moved == (knob is None and mode == dn.MODE_TF32 and tail == "yolo"), net.layer_describe(2)
        net.close()
    for a, b in zip(*out):
        if mode == dn.MODE_TF32 and tail == "yolo":
            parity(a, b, 1e-2)
        else:
            assert np.array_equal(a, b)


@pytest.mark.parametrize("mode", [dn.MODE_TF32, dn.MODE_BF16])
def test_parts_of_a_batch_keep_its_kernels(mode, tmp_path, monkeypatch):
    """A step that runs in parts, first layers and last ones with plans of their own over fewer images: those plans choose between the kernels whose sums run in
    different orders as the whole batch's does, and the results are its, to the bit."""
    import numpy as np
    import torch
    from darknet_b200 import synth
    monkeypatch.delenv("DNB_TC_TAPS", raising=False)
    cfg = (synth._net(16, 256, 256) + synth._conv(32, 3) + synth._conv(64, 3, stride=2) + synth._conv(128, 3) + synth._conv(64, 1) + synth._conv(128, 3) + synth._conv(128, 3) +
           synth._conv(90, 1, bn=False, act="linear") + synth._yolo("0,1", "10,14, 23,27", 2, 40))
    path = str(tmp_path / "b.weights")
    synth.write_weights(path, synth.seeded_params(cfg, 27))
    x = synth.seeded_input(cfg, 28)
    whole, parts = (dn.Network(cfg, path, mode, text=True) for _ in range(2))
    whole.forward(torch.from_numpy(x).cuda())
    torch.cuda.synchronize()
    got = parts.predict(x)
    tiles = lambda net, i: net.layer_describe(i).split("tiles=")[1].split()[0]  # noqa: E731
    for i in (2, 4):
        assert "one_load_for_nine_taps" in whole.layer_describe(i) and "one_load_for_nine_taps" in parts.layer_describe(i), i
    assert int(tiles(parts, 2)) < int(tiles(whole, 2))
    assert np.array_equal(got.reshape(-1), whole.layer_output(7).reshape(-1))
    whole.close(), parts.close()


@pytest.mark.parametrize("mode,batch,c,n,height,width,layout,taken", [
    (dn.MODE_TF32, 2, 96, 96, 239, 210, "nhwc", True), (dn.MODE_TF32, 2, 40, 96, 260, 104, "nhwc", True), (dn.MODE_BF16, 2, 96, 96, 112, 229, "nhwc", True),
    (dn.MODE_BF16, 2, 128, 96, 126, 224, "nhwc", True), (dn.MODE_TF32, 4, 512, 1024, 19, 19, "nhwc", True), (dn.MODE_TF32, 8, 256, 512, 52, 52, "nchw", True),
    (dn.MODE_TF32, 2, 96, 128, 76, 75, "nhwc", False), (dn.MODE_TF32, 2, 64, 64, 152, 152, "nhwc", False), (dn.MODE_BF16, 2, 128, 256, 38, 38, "nhwc", False),
    (dn.MODE_TF32, 2, 256, 96, 100, 90, "nhwc", False)])
def test_layers_that_take_one_load_for_nine_taps_by_themselves(mode, batch, c, n, height, width, layout, taken, monkeypatch):
    """The choice as it is without a knob.  Two images take what one takes, and an image's result is the same, to the bit; whole numbers are what they are without the kernel."""
    import numpy as np
    for knob in ("DNB_TC_TAPS", "DNB_TC_SPLITK", "DNB_TC_PAIR"):
        monkeypatch.delenv(knob, raising=False)
    case = conv_case(785, b=batch, c=c, h=height, w=width, n=n, size=3, bn=False)
    plan, whole, _ = run_conv(case, mode, "nhwc", layout)
    assert ("one_load_for_nine_taps" in plan.describe()) == taken, plan.describe()
    if batch == 2:
        for k in range(2):
            alone, one, _ = run_conv(dict(case, x=case["x"][k:k + 1]), mode, "nhwc", layout)
            assert ("one_load" in alone.describe()) == taken and np.array_equal(one[0], whole[k]), alone.describe()
    case = dict(case, x=np.rint(2 * case["x"]), w=np.rint(case["w"] / np.abs(case["w"]).max() * 6), biases=np.rint(9 * case["biases"]))
    out = [run_conv(case, mode, "nhwc", layout)[1]]
    monkeypatch.setenv("DNB_TC_TAPS", "0")
    out.append(run_conv(case, mode, "nhwc", layout)[1])
    assert np.array_equal(*out)


def test_calls_go_to_the_current_stream():
    """Inside torch's stream contexts, nested and left again, and to the stream that the caller names."""
    import torch
    from darknet_b200.api import _stream
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        assert _stream().value == a.cuda_stream
        with torch.cuda.stream(b):
            assert _stream().value == b.cuda_stream and _stream(a.cuda_stream).value == a.cuda_stream
        assert _stream().value == a.cuda_stream
    assert (_stream().value or 0) == torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("channels,height,width", [(32, 1, 1), (33, 1, 7), (127, 3, 3), (128, 8, 1), (129, 7, 7), (260, 8, 8), (1000, 13, 5), (100, 23, 27), (6000, 5, 2)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_global_average_keeps_its_order(channels, height, width, dtype):
    """Row j adds pixels j, j + 8, ...; the eight rows are added in order and divided by the pixels: equal to the bit to that, and channels
    of a wider map that are not the tensor's stay out of it."""
    import numpy as np
    import torch
    dt, batch = getattr(torch, dtype), 5 if channels > 2000 else 3
    pitch = (channels + 7) // 8 * 8 + 8
    full = torch.randn((batch, height, width, pitch), generator=torch.Generator().manual_seed(channels)).to(dt)
    rows = full[..., :channels].float().numpy().reshape(batch, height * width, channels)
    want = np.zeros((batch, channels), np.float32)
    for j in range(8):
        row = np.zeros((batch, channels), np.float32)
        for p in range(j, height * width, 8):
            row += rows[:, p]
        want += row
    want = torch.from_numpy(want / np.float32(height * width)).to(dt).float().numpy()
    x, y = full.cuda(), torch.full((batch, 1, 1, pitch), -7.0, dtype=dt, device="cuda")
    dn.avgpool(dn.as_tensor(x, dn.NHWC, channels), dn.as_tensor(y, dn.NHWC, channels))
    torch.cuda.synchronize()
    got = y.float().cpu().numpy()[:, 0, 0]
    assert np.array_equal(got[:, :channels], want) and (got[:, channels:] == -7.0).all()


@pytest.mark.parametrize("odd", ["bias", "pixel"])
@pytest.mark.parametrize("channels", [1, 3])
def test_a_first_layers_tiles_keep_to_themselves(odd, channels, tmp_path, monkeypatch):
    """More tiles than CTAs at once: an infinite value of one tile changes nothing in the tiles that the same CTA does after it.  As in two launches, to the bit."""
    import numpy as np
    from darknet_b200 import synth
    batch, size = 8, 224                                     # 784 tiles; four CTAs an SM are 592
    cfg = (synth._net(batch, size, size, channels) + synth._conv(32, 3) + "\n[maxpool]\nsize=2\nstride=2\n" + synth._conv(32, 3, xnor=True) + "\n[avgpool]\n")
    params = synth.seeded_params(cfg, 23)
    x = synth.seeded_input(cfg, 24, "normal")
    if odd == "bias":
        params[0].biases[31] = np.inf
    else:
        params[0].weights[28:] = np.abs(params[0].weights[28:])
        x[:4, 0, 10::64, 10::32] = np.inf
    path = str(tmp_path / "i.weights")
    synth.write_weights(path, params)
    out = []
    for fuse in ("0", "1"):
        monkeypatch.setenv("DNB_FUSE_POOL", fuse)
        net = dn.Network(cfg, path, dn.MODE_TF32, text=True)
        net.predict(x)
        out.append([net.layer_output(i) for i in (1, 2)] + [net.launches])
        net.close()
    assert out[1][-1] < out[0][-1] and np.isinf(out[0][0]).any()
    for a, b in zip(out[0][:-1], out[1][:-1]):
        assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("odd", ["zeros", "nan_bias", "scales", "pixels"])
@pytest.mark.parametrize("batch,size", [(2, 88), (3, 36)])     # maps that end inside a tile of 16 x 8 windows, both ways
def test_signs_of_a_first_layer_with_its_maxpool(odd, batch, size, tmp_path, monkeypatch):
    """What the next xnor layer makes of values that are -0, infinite or NaN before they are rounded: as in two launches, to the bit.  A zero
    sum of a filter with a negative scale and a bias of -0 is -0, and so is a NaN or a tiny negative value once it is rounded to TF32."""
    import numpy as np
    from darknet_b200 import synth
    cfg = (synth._net(batch, size, size) + synth._conv(32, 3) + "\n[maxpool]\nsize=2\nstride=2\n" + synth._conv(48, 3, xnor=True) + "\n[avgpool]\n")
    params = synth.seeded_params(cfg, 21)
    x = synth.seeded_input(cfg, 22, "normal")
    first = params[0]
    first.rolling_mean[:] = 0
    first.biases[:8] = -0.0
    first.scales[:32:2] *= -1
    first.biases[8:12] = -1e-42
    x[:, :, size // 3:] = 0
    if odd == "nan_bias":
        first.biases[[0, 5, 31]] = np.nan
        first.biases[[1, 30]] = np.inf, -np.inf
    if odd == "scales":
        first.scales[[2, 9, 28]] = 0.0, -0.0, np.nan
    if odd == "pixels":
        x[0, 0, 8, 6], x[0, 1, size - 2, 2], x[-1, 2, 4, size - 2] = np.nan, np.inf, -np.inf
    path = str(tmp_path / "s.weights")
    synth.write_weights(path, params)
    out = []
    for fuse in ("0", "1"):
        monkeypatch.setenv("DNB_FUSE_POOL", fuse)
        net = dn.Network(cfg, path, dn.MODE_TF32, text=True)
        net.predict(x)
        out.append([net.layer_output(i) for i in (1, 2)] + [net.launches])
        net.close()
    assert out[1][-1] < out[0][-1]
    for a, b in zip(out[0][:-1], out[1][:-1]):
        assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("mode", [dn.MODE_TF32, dn.MODE_BF16])
def test_one_plan_several_epilogues(mode, monkeypatch):
    """One plan and its tensors, called with one epilogue after another, each of which another kernel may have to do: as a new plan does each, to the bit."""
    import ctypes as C
    import numpy as np
    import torch
    from gpu_util import dev_nhwc, empty_nchw, empty_nhwc
    monkeypatch.setenv("DNB_TC_TAPS", "2")
    store = torch.bfloat16 if mode == dn.MODE_BF16 else torch.float32
    case = conv_case(780, b=3, c=64, h=15, w=14, n=96, size=3)
    xt, xd = dev_nhwc(case["x"], store)
    at, ad = dev_nhwc(np.random.Generator(np.random.Philox(key=[8, 9])).standard_normal((3, 96, 15, 14), dtype=np.float32), store)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def plan_of(act):
        p = dn.ConvPlan(3, 64, 15, 14, 96, 3, 1, 1, 1, True, act, False, mode)
        p.set_params(case["w"], case["biases"], case["scales"], case["mean"], case["var"])
        return p

    def call(plan, what, yt, yd):
        if what == "forward":
            plan.forward(xd, yd)
        elif what == "yolo":
            dn.check(dn.lib().dnb_conv_yolo_forward(plan.handle, C.byref(xd), C.byref(yd), 3, 27, stream))
        else:
            dn.check(dn.lib().dnb_conv_shortcut_forward(plan.handle, C.byref(xd), C.byref(ad), C.byref(yd), 1.0, 1.0, dn.ACTIVATIONS[what], stream))
        torch.cuda.synchronize()
        plan.check_status()
        return yt.float().cpu().numpy()

    for act, empty, calls in (("leaky", lambda: empty_nhwc(3, 96, 15, 14, store), ["linear", "leaky", "relu", "linear", "forward", "leaky"]),
                              ("linear", lambda: empty_nchw(3, 96, 15, 14), ["forward", "yolo", "forward", "yolo"])):
        yt, yd = empty()
        plan = plan_of(act)
        for what in calls:
            got = call(plan, what, yt, yd)
            assert np.array_equal(got, call(plan_of(act), what, *empty())), (act, what)
