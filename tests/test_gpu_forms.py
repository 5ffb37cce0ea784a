"""GPU parity of the forms that launch plans choose by size, type and value range, at the edges of their ranges."""
import numpy as np
import pytest

from oracle import graph_runner
from tpu_compiler_b200 import graphs

pytestmark = pytest.mark.gpu


def has_form(m, name, **words):
    form = m.op_form(name)
    return all(form.get(k) == v for k, v in words.items())


def run_model(text, weights, inputs, names, **form):
    from tpu_compiler_b200 import module
    m = module(0)
    m.load_text(text, weights)
    assert has_form(m, names[0], **form), m.op_form(names[0])
    for k, v in inputs.items():
        m.set_tensor(k, v)
    m.invoke()
    ref = graph_runner.run(text, weights, inputs)
    out = {n: (m.get_tensor(n), ref[n]) for n in names}
    m.close()
    return out


def conv_text(dtype, n, ic, oc, hw, k, s, p, d, relu, int8=False, extra=""):
    o = (hw + 2 * p - d * (k - 1) - 1) // s + 1
    return ("conv_2d name=c in=x,f,b%s shape=%d,%d,%d,%d dtype=%s kh=%d kw=%d sh=%d sw=%d pt=%d pb=%d pl=%d pr=%d dh=%d dw=%d g=1 "
            "do_relu=%d with_bias=1%s\n" % (",-,-,r,m" if int8 else "", n, oc, o, o, dtype, k, k, s, s, p, p, p, p, d, d, relu, extra))


@pytest.mark.parametrize("relu", [False, True])
@pytest.mark.parametrize("mults", ["normalised", "large_powers", "random", "power_of_two", "small"])
def test_float_requantisation_edges(relu, mults):
    """Every shift of the floating-point form's range, normalised multipliers and those that make exact ties in the first rounding
    (powers of two); with zero multipliers or ones of few significant bits, whose addend is no float, the same layers on the integer
    form (with ReLU) and the 64-bit one (shifts of 30 and 31)."""
    rng = np.random.default_rng(5 + relu)
    ic, oc, hw = 32, 96, 12
    f = rng.integers(-20, 21, (oc, ic, 1, 1)).astype(np.float32)
    r = (np.arange(oc) % (23 if relu else 32)).astype(np.float32)
    m = {"random": (rng.integers(2 ** 23, 2 ** 24, oc) * 128).astype(np.float32),
         "power_of_two": np.float32(2.0) ** rng.integers(7, 31, oc).astype(np.float32),
         "small": (rng.integers(0, 64, oc) * 2 ** 20).astype(np.float32),
         "normalised": (rng.integers(2 ** 23, 2 ** 24, oc) * 128).astype(np.float32),
         "large_powers": np.float32(2.0) ** np.where(r < 22, rng.integers(29, 31, oc), 30).astype(np.float32)}[mults]
    floating = mults in ("normalised", "large_powers")
    if not floating:
        m[::17] = 0
    b = rng.integers(-2 ** 18, 2 ** 18, oc).astype(np.float32)
    b[:23] = rng.integers(-3, 4, 23)  # small sums around zero at every shift
    text = "input name=x shape=2,%d,%d,%d dtype=INT8\n" % (ic, hw, hw) + conv_text("INT8", 2, ic, oc, hw, 1, 1, 0, 1, int(relu), True)
    x = rng.integers(-128, 128, (2, ic, hw, hw)).astype(np.float32)
    got, ref = run_model(text, {"f": f, "b": b, "r": r, "m": m}, {"x": x}, ["c"],
                         requant="float" if floating else ("integer" if relu else "wide"))["c"]
    assert np.array_equal(got, ref)


WINDOWS = [  # n, ic, oc, hw, k, stride, pad, dilation: pixel groups of 4, 2 and 1, tile remainders, 16-byte pixels
    (2, 3, 32, 36, 3, 1, 1, 1), (1, 3, 24, 34, 3, 2, 1, 1), (3, 3, 64, 30, 7, 2, 3, 1), (1, 3, 64, 31, 5, 2, 2, 1),
    (2, 4, 100, 18, 3, 1, 1, 2), (1, 1, 16, 9, 3, 1, 1, 1), (2, 2, 40, 26, 4, 2, 1, 1), (1, 3, 16, 17, 3, 4, 0, 1)]


@pytest.mark.parametrize("case", WINDOWS + [(2, 12, 48, 20, 3, 1, 1, 1), (1, 7, 64, 24, 5, 2, 2, 1)])
@pytest.mark.parametrize("shared", [False, True])  # True: another consumer of the input keeps it from the window layout
def test_row_window_conv_i8(case, shared):
    n, ic, oc, hw, k, s, p, d = case
    model = graphs.single_conv_i8(n, ic, oc, hw, k, s, p, d, seed=3100 + ic + k)
    text = model.text + ("relu name=other in=x shape=%d,%d,%d,%d dtype=INT8\n" % (n, ic, hw, hw) if shared else "")
    for name, (got, ref) in run_model(text, model.weights, {"x": model.meta["x"]}, ["conv"] + ["other"] * shared + ["x"]).items():
        assert np.array_equal(got, ref), name


@pytest.mark.parametrize("dtype", ["BF16", "FP32"])
@pytest.mark.parametrize("case", WINDOWS)
def test_row_window_conv_float(dtype, case):
    n, ic, oc, hw, k, s, p, d = case
    rng = np.random.default_rng(41 + ic + k)
    cut = graphs._bf16_np if dtype == "BF16" else (lambda v: np.asarray(v, np.float32))
    w = {"f": cut(rng.normal(0, 0.2, (oc, ic, k, k))), "b": rng.normal(0, 0.2, oc).astype(np.float32)}
    x = cut(rng.normal(0, 1, (n, ic, hw, hw)))
    text = "input name=x shape=%d,%d,%d,%d dtype=%s\n" % (n, ic, hw, hw, dtype) + conv_text(dtype, n, ic, oc, hw, k, s, p, d, 1)
    got, ref = run_model(text, w, {"x": x}, ["c"])["c"]
    if dtype == "BF16":
        assert np.all(np.abs(got - ref) <= np.maximum(np.abs(ref) * 2.0 ** -7, 2.0 ** -8 * np.abs(ref).max() * 2.0 ** -6))
    else:
        assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("dtype", ["INT8", "BF16", "FP32"])
@pytest.mark.parametrize("case", [
    # n, ic, oc, hw, k, stride, pad, dilation
    (3, 64, 64, 14, 3, 1, 1, 1),    # pixel pairs, steps of K skipped at both ends
    (2, 32, 32, 10, 5, 1, 2, 1), (1, 48, 24, 12, 3, 1, 0, 1), (2, 64, 48, 12, 3, 1, 2, 2),  # pairs: other filters, pads
    (2, 16, 16, 20, 1, 1, 0, 1), (3, 96, 40, 6, 1, 1, 0, 1),  # pairs twice; pairs of a 1x1 with a long K
    (5, 128, 96, 7, 3, 1, 1, 1),    # several images per tile
    (2, 40, 136, 13, 3, 1, 2, 2), (1, 64, 130, 31, 3, 1, 1, 1), (1, 72, 80, 57, 5, 1, 1, 1),  # odd extents, ragged tiles
    (1, 512, 64, 9, 3, 1, 1, 1), (1, 256, 200, 5, 1, 1, 0, 1),  # few tiles and a long K
    (2, 80, 64, 13, 3, 2, 1, 1), (7, 72, 72, 12, 5, 1, 2, 1), (2, 144, 160, 9, 3, 1, 1, 1),  # channels off the sector grid
    (1, 64, 256, 55, 1, 1, 0, 1), (1, 64, 256, 56, 1, 1, 0, 1),  # the last half tiles and the first whole ones (148 SMs)
    (2, 64, 96, 11, 3, 2, 1, 1)])   # a stride
def test_conv_forms(dtype, case):
    n, ic, oc, hw, k, s, p, d = case
    if dtype == "INT8":
        model = graphs.single_conv_i8(n, ic, oc, hw, k, s, p, d, seed=5200 + ic + k)
        got, ref = run_model(model.text, model.weights, {"x": model.meta["x"]}, ["conv"])["conv"]
        assert np.array_equal(got, ref)
        return
    rng = np.random.default_rng(43 + ic + k)
    cut = graphs._bf16_np if dtype == "BF16" else (lambda v: np.asarray(v, np.float32))
    w = {"f": cut(rng.normal(0, (2.0 / (ic * k * k)) ** 0.5, (oc, ic, k, k))), "b": rng.normal(0, 0.2, oc).astype(np.float32)}
    x = cut(rng.normal(0, 1, (n, ic, hw, hw)))
    text = "input name=x shape=%d,%d,%d,%d dtype=%s\n" % (n, ic, hw, hw, dtype) + conv_text(dtype, n, ic, oc, hw, k, s, p, d, 1)
    got, ref = run_model(text, w, {"x": x}, ["c"])["c"]
    if dtype == "BF16":
        assert np.all(np.abs(got - ref) <= np.maximum(np.abs(ref) * 2.0 ** -7, 2.0 ** -14 * np.abs(ref).max()))
    else:
        assert np.abs(got - ref).max() <= 3e-5 * np.abs(ref).max()


@pytest.mark.parametrize("graph", [1, 0])
def test_large_result_read_before_the_end(graph):
    """A large result that ends before the module does is fetched beside the ops behind it: launch after launch, each with
    inputs of its own, in any order of fetching, and behind something else than a launch."""
    from tpu_compiler_b200 import module
    rng = np.random.default_rng(9)
    text = ("input name=x shape=4,64,64,64 dtype=INT8\n"
            "relu name=early in=x shape=4,64,64,64 dtype=INT8\n"  # 4 MB as fp32, nothing reads it
            "pool_max_2d name=p in=x shape=4,64,64,64 dtype=INT8 kh=3 kw=3 sh=1 sw=1 pt=1 pb=1 pl=1 pr=1\n"
            "pool_max_2d name=q in=p shape=4,64,32,32 dtype=INT8 kh=2 kw=2 sh=2 sw=2 pt=0 pb=0 pl=0 pr=0\n"
            "relu name=late in=q shape=4,64,32,32 dtype=INT8\n")
    m = module(0)
    m.load_text(text, {})
    m.set_option("cuda_graph", graph)
    for i in range(8):
        x = rng.integers(-128, 128, (4, 64, 64, 64)).astype(np.float32)
        m.set_tensor("x", x)
        m.launch()
        if i == 5:
            m.set_tensor("x", -x - 1)  # the launch in flight keeps its input
        ref = graph_runner.run(text, {}, {"x": x})
        for name in (["early", "late", "early"], ["late", "early", "p"])[i % 2]:
            assert np.array_equal(m.get_tensor(name), ref[name]), (i, name)
    m.close()


@pytest.mark.parametrize("dtype", ["INT8", "BF16"])
@pytest.mark.parametrize("case", [  # n, c, hw, k, stride, pad, out
    (2, 48, 17, 3, 2, 1, 9), (1, 16, 16, 3, 2, 0, 8), (2, 40, 13, 3, 1, 1, 13), (1, 16, 5, 2, 2, 0, 3), (3, 32, 8, 2, 2, 1, 5),  # strips
    (2, 16, 13, 13, 1, 6, 13), (1, 80, 13, 9, 1, 4, 13), (2, 64, 7, 5, 1, 2, 7), (1, 32, 28, 7, 1, 3, 28),  # planes, the last too large for one
    (1, 32, 9, 4, 3, 1, 3), (2, 32, 6, 3, 3, 0, 2)])  # any window
def test_max_pool_forms(dtype, case):
    n, c, hw, k, s, p, o = case
    rng = np.random.default_rng(60 + hw + k)
    x = rng.integers(-128, 128, (n, c, hw, hw)).astype(np.float32) if dtype == "INT8" else graphs._bf16_np(rng.normal(0, 3, (n, c, hw, hw)))
    text = ("input name=x shape=%d,%d,%d,%d dtype=%s\npool_max_2d name=p in=x shape=%d,%d,%d,%d dtype=%s kh=%d kw=%d sh=%d sw=%d pt=%d pb=%d "
            "pl=%d pr=%d\n" % (n, c, hw, hw, dtype, n, c, o, o, dtype, k, k, s, s, p, p, p, p))
    got, ref = run_model(text, {}, {"x": x}, ["p"])["p"]
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("channels", [[16, 48], [32], [16] * 8, [16, 32, 16, 16, 48, 16, 16, 64, 32]])
def test_concat_in_one_launch(channels):
    rng = np.random.default_rng(len(channels))
    shapes = ["input name=x%d shape=2,%d,5,7 dtype=INT8\n" % (i, c) for i, c in enumerate(channels)]
    names = ["x%d" % i for i in range(len(channels))]
    w = {"r": (7 * (np.arange(len(channels)) % 2)).astype(np.float32), "m": np.where(np.arange(len(channels)) % 2, 90, 1).astype(np.float32)}
    text = "".join(shapes) + "concat name=y in=%s,-,-,r,m shape=2,%d,5,7 dtype=INT8 axis=1 do_relu=0\n" % (",".join(names), sum(channels))
    x = {nm: rng.integers(-128, 128, (2, c, 5, 7)).astype(np.float32) for nm, c in zip(names, channels)}
    got, ref = run_model(text, w, x, ["y"])["y"]
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("dtype", ["INT8", "BF16"])
def test_upsample_vectors(dtype):
    x = np.random.default_rng(2).integers(-128, 128, (2, 48, 5, 6)).astype(np.float32)
    text = "input name=x shape=2,48,5,6 dtype=%s\nupsample name=u in=x shape=2,48,15,12 dtype=%s scale_h=3 scale_w=2\n" % (dtype, dtype)
    got, ref = run_model(text, {}, {"x": x}, ["u"])["u"]
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("count", [1, 2, 3, 4])
def test_bf16_add_operand_counts(count):
    rng = np.random.default_rng(count)
    names = ["x%d" % i for i in range(count)]
    text = "".join("input name=%s shape=3,24,9,11 dtype=BF16\n" % nm for nm in names)
    text += "eltwise_add name=y in=%s shape=3,24,9,11 dtype=BF16 do_relu=1\n" % ",".join(names)
    x = {nm: graphs._bf16_np(rng.normal(0, 2, (3, 24, 9, 11))) for nm in names}
    got, ref = run_model(text, {}, x, ["y"])["y"]
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("relu", [0, 1])
@pytest.mark.parametrize("case", [(1, 16, 9, 1), (2, 32, 7, 2), (32, 192, 15, 1), (40, 192, 21, 2)])  # n, c, hw, stride: one row, two rows
@pytest.mark.parametrize("wide", [False, True])  # True: a channel outside the floating-point requantisation
def test_depthwise_rows_and_requantisation(relu, case, wide):
    n, c, hw, s = case
    rng = np.random.default_rng(c + hw)
    o = (hw - 1) // s + 1
    w = {"f": rng.integers(-127, 128, (c, 1, 3, 3)).astype(np.float32), "b": rng.integers(-5000, 5000, c).astype(np.float32),
         "r": rng.integers(6, 11, c).astype(np.float32), "m": (rng.integers(2 ** 23, 2 ** 24, c) * 128).astype(np.float32)}
    if wide:
        w["b"][3], w["r"][3] = 2.0 ** 24, 18  # sums past its range, and a shift whose results there are not all saturated
    x = rng.integers(-128, 128, (n, c, hw, hw)).astype(np.float32)
    text = ("input name=x shape=%d,%d,%d,%d dtype=INT8\nconv_2d name=c in=x,f,b,-,-,r,m shape=%d,%d,%d,%d dtype=INT8 kh=3 kw=3 sh=%d sw=%d "
            "pt=1 pb=1 pl=1 pr=1 dh=1 dw=1 g=%d do_relu=%d with_bias=1\n" % (n, c, hw, hw, n, c, o, o, s, s, c, relu))
    got, ref = run_model(text, w, {"x": x}, ["c"], tiles="depthwise", requant="integer" if wide else "float")["c"]
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("case", [(13, 64, 256, 30, 2), (9, 64, 200, 21, 1), (3, 128, 144, 15, 1), (40, 16, 272, 13, 1)])  # n, ic, oc, hw, mode
def test_residual_add_with_prefetch(case):
    """Fused adds over several tiles per CTA, ragged tiles and channel tiles that some warps have no part in."""
    from tpu_compiler_b200 import module
    n, ic, oc, hw, mode = case
    rng = np.random.default_rng(oc)
    model = graphs.single_conv_i8(n, ic, oc, hw, 1, 1, 0, relu=False, seed=77)
    w = dict(model.weights, ar=np.array([7.0], np.float32), am=np.array([70.0, 60.0], np.float32))
    shape = "shape=%d,%d,%d,%d dtype=INT8" % (n, oc, hw, hw)
    text = "input name=res %s\n" % shape + model.text + "eltwise_add name=s in=res,conv,-,-,ar,am %s do_relu=1\n" % shape
    x = {"x": model.meta["x"], "res": rng.integers(-128, 128, (n, oc, hw, hw)).astype(np.float32)}
    ref = graph_runner.run(text, w, x)
    m = module(0)
    m.set_option("fuse_residual_add", mode)
    m.load_text(text, w)
    assert m.kernel_count() == 1
    for name, v in x.items():
        m.set_tensor(name, v)
    for _ in range(2):
        m.invoke()
    assert all(np.array_equal(m.get_tensor(k), ref[k]) for k in ("conv", "s"))
    m.close()


@pytest.mark.parametrize("case", [  # n, ic, oc, hw, big_tiles, fuse_residual_add
    (16, 64, 128, 56, 1, 1), (2, 96, 136, 13, 1256, 1), (2, 96, 136, 13, 2192, 1),   # every add: large tiles by size, and forced on a small layer
    (32, 64, 128, 56, 1, 2), (97, 256, 512, 14, 1, 2)])                             # by size: 9 and 18 K blocks of a layer that widens
def test_adds_behind_layers_that_fill_the_gpu(case):
    """Layers that would run large tiles do not when their add is fused: it launches nothing, both tensors keep their bits."""
    from tpu_compiler_b200 import module
    n, ic, oc, hw, big, mode = case
    model = graphs.single_conv_i8(1, ic, oc, hw, 3, 1, 1, relu=False, seed=78)
    w = dict(model.weights, ar=np.array([7.0], np.float32), am=np.array([70.0, 60.0], np.float32))
    shape = "shape=%d,%d,%d,%d dtype=INT8" % (n, oc, hw, hw)
    text = ("input name=res %s\n" % shape + model.text.replace("shape=1,", "shape=%d," % n) +
            "eltwise_add name=s in=res,conv,-,-,ar,am %s do_relu=1\n" % shape)
    rng = np.random.default_rng(oc)
    x = {"x": rng.integers(-128, 128, (n, ic, hw, hw)).astype(np.float32), "res": rng.integers(-128, 128, (n, oc, hw, hw)).astype(np.float32)}
    got = []
    for fuse in (0, mode):
        m = module(0)
        m.set_option("fuse_residual_add", fuse)
        m.set_option("big_tiles", big)
        m.load_text(text, w)
        for name, v in x.items():
            m.set_tensor(name, v)
        m.invoke()
        got.append([m.get_tensor(k) for k in ("conv", "s")] + [m.kernel_count()])
        m.close()
    assert got[1][2] == got[0][2] - 1
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("dtype", ["INT8", "BF16", "FP32"])
@pytest.mark.parametrize("shape", [
    (1, 1, 1, 1), (3, 1001, 1, 1), (5, 3, 17, 23), (2, 70, 9, 5),        # value by value, small results into pinned memory
    (1, 32, 181, 181), (1, 32, 181, 182), (1, 31, 190, 190), (2, 33, 130, 130), (1, 2048, 23, 23),  # both sides of 2^20 values, 32 channels
    (1, 4194305, 1, 1)])                                               # more channels than a grid has rows of tiles
def test_download_forms(dtype, shape):
    from tpu_compiler_b200 import module
    if dtype != "INT8" and shape[1] > 10 ** 6:
        pytest.skip("one type is enough")
    m = module(0)
    m.load_text("input name=x shape=%d,%d,%d,%d dtype=%s\n" % (shape + (dtype,)), {})
    x = np.random.default_rng(sum(shape)).integers(-128, 128, shape).astype(np.float32)
    m.set_tensor("x", x)
    assert np.array_equal(m.get_tensor("x"), x)
    m.close()


@pytest.mark.parametrize("case", [  # n, ic, oc, hw, k, pixels per tile, parts (148 SMs)
    (11, 512, 512, 7, 3, 64, 4), (12, 512, 512, 7, 3, 64, 1),  # 36 K blocks: the most tiles that are still split, the fewest that are not
    (15, 1024, 512, 7, 3, 64, 3), (23, 1024, 512, 7, 3, 64, 2), (24, 1024, 512, 7, 3, 64, 1),  # 72: in three, in two, not
    (8, 512, 512, 7, 3, 64, 5), (3, 330, 520, 8, 5, 64, 9), (1, 330, 200, 6, 5, 64, 11),        # a last part of fewer K blocks
    (25, 330, 512, 8, 5, 128, 2), (36, 330, 512, 8, 5, 128, 2), (37, 330, 512, 8, 5, 128, 1)])  # 75: tiles of 128 pixels, whose blocks are shared, too
def test_split_rule_edges(case):
    from tpu_compiler_b200 import module
    n, ic, oc, hw, k, pixels, parts = case
    model = graphs.single_conv_i8(n, ic, oc, hw, k, 1, k // 2, relu=parts % 2 == 0, seed=3300 + k)
    got = []
    for split in (1, 0):
        m = module(0)
        m.set_option("split_k", split)
        m.load_text(model.text, model.weights)
        assert has_form(m, "conv", tiles="small", pixels=pixels, split_k=parts if split else 1), m.op_form("conv")
        m.set_tensor("x", model.meta["x"])
        for _ in range(2):
            m.invoke()
            got.append(m.get_tensor("conv"))
        m.close()
    assert all(np.array_equal(g, got[-1]) for g in got)


@pytest.mark.parametrize("relu", [0, 1])
def test_bf16_results_past_the_largest_finite(relu):
    """Sums that overflow or round past the largest BF16 become +0x7f7f for either sign; ReLU makes negative ones zero. Every
    product is exact; channels and pixels leave remainders of a 32 x 32 block."""
    rng = np.random.default_rng(11)
    n, ic, oc, hw = 2, 32, 40, 9
    f = np.zeros((oc, ic, 1, 1), np.float32)
    f[np.arange(oc), np.arange(oc) % ic, 0, 0] = np.where(np.arange(oc) % 3 == 2, -1, 1) * np.float32(2.0) ** np.where(np.arange(oc) % 2, 64, 0)
    x = np.float32(2.0) ** 63 * rng.choice([-3.0, -1.9921875, -1.0, 0.0, 1.0, 1.9921875, 3.0], (n, ic, hw, hw)).astype(np.float32)
    b = np.where(np.arange(oc) % 5 == 0, 2.0 ** 119, 0.0).astype(np.float32)  # half of the last place of the largest finite value
    text = "input name=x shape=%d,%d,%d,%d dtype=BF16\n" % (n, ic, hw, hw) + conv_text("BF16", n, ic, oc, hw, 1, 1, 0, 1, relu)
    got, ref = run_model(text, {"f": f, "b": b}, {"x": x}, ["c"])["c"]
    assert (ref == graphs._bf16_np(np.float32(3.39e38))).any()
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("dtype", ["INT8", "BF16", "FP32"])
@pytest.mark.parametrize("form", [1256, 1096, 2256, 2192, 2032])  # 1000 CTAs per tile + pixels per tile
@pytest.mark.parametrize("case", [
    # n, ic, oc, hw, k, stride, pad, dilation, ReLU
    (3, 64, 256, 20, 1, 1, 0, 1, 0),    # one short K block, the last tile's second half past the last pixel
    (2, 96, 136, 13, 3, 1, 1, 1, 1),    # channels that end inside a tile, K blocks with a tail
    (5, 160, 300, 9, 3, 2, 1, 1, 0),    # a stride, images inside a tile
    (1, 1040, 520, 5, 1, 1, 0, 1, 1),   # fewer pixels than a tile, a long K, a channel tile that one CTA of a pair has alone
    (23, 80, 144, 41, 3, 1, 1, 1, 0)])  # several tiles per CTA
def test_big_tiles(dtype, form, case):
    from tpu_compiler_b200 import module
    n, ic, oc, hw, k, s, p, d, relu = case
    if dtype == "FP32":
        oc = (oc + 15) // 16 * 16  # (their channels are padded to 4 only, and large tiles take whole sixteens)
    if dtype == "INT8":
        model = graphs.single_conv_i8(n, ic, oc, hw, k, s, p, d, relu=bool(relu), seed=6200 + ic + k)
        text, w, x, name = model.text, model.weights, model.meta["x"], "conv"
    else:
        rng = np.random.default_rng(47 + ic + k)
        cut = graphs._bf16_np if dtype == "BF16" else (lambda v: np.asarray(v, np.float32))
        w = {"f": cut(rng.normal(0, (2.0 / (ic * k * k)) ** 0.5, (oc, ic, k, k))), "b": rng.normal(0, 0.2, oc).astype(np.float32)}
        x, name = cut(rng.normal(0, 1, (n, ic, hw, hw))), "c"
        text = "input name=x shape=%d,%d,%d,%d dtype=%s\n" % (n, ic, hw, hw, dtype) + conv_text(dtype, n, ic, oc, hw, k, s, p, d, relu)
    got = []
    for mode in (0, form):
        m = module(0)
        m.set_option("big_tiles", mode)
        m.load_text(text, w)
        assert has_form(m, name, **(dict(tiles="big", ctas=form // 1000, pixels=form % 1000) if mode else dict(tiles="small"))), m.op_form(name)
        m.set_tensor("x", x)
        for _ in range(2):
            m.invoke()
        got.append(m.get_tensor(name))
        m.close()
    # the products of an output value are summed in the same order: every bit is the same
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("relu", [0, 1])
@pytest.mark.parametrize("case", [  # n, ic, oc, hw, k, stride, pad, dilation: the patches built in shared memory
    (1, 3, 16, 9, 3, 1, 1, 1),      # fewer tiles than SMs, an odd number of taps
    (3, 3, 64, 65, 7, 2, 3, 1),     # ragged last tile
    (2, 4, 40, 64, 6, 3, 2, 1),     # an even number of taps, four channels, channels that end inside a quarter
    (5, 1, 64, 96, 7, 1, 6, 2),     # several tiles per SM, a dilation, taps outside the image
    (1, 3, 64, 30, 8, 2, 3, 1), (1, 3, 72, 30, 7, 2, 3, 1)])  # too many taps, too many channels: the patch matrix
def test_fp32_stem_patches(case, relu):
    n, ic, oc, hw, k, s, p, d = case
    rng = np.random.default_rng(53 + oc + k)
    w = {"f": rng.normal(0, (2.0 / (ic * k * k)) ** 0.5, (oc, ic, k, k)).astype(np.float32), "b": rng.normal(0, 0.2, oc).astype(np.float32)}
    x = rng.normal(0, 1, (n, ic, hw, hw)).astype(np.float32)
    text = "input name=x shape=%d,%d,%d,%d dtype=FP32\n" % (n, ic, hw, hw) + conv_text("FP32", n, ic, oc, hw, k, s, p, d, relu)
    got, ref = run_model(text, w, {"x": x}, ["c"])["c"]
    # three products leave 2^-22 of each term; the tensor core cuts each of the 25 partial sums of a term at 2^-23 of the sum
    assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("case", [(13, 64, 256, 30, 1), (9, 64, 200, 21, 1), (3, 128, 144, 15, 1), (40, 16, 272, 13, 1), (64, 64, 256, 20, 2)])  # n, ic, oc, hw, mode
def test_bf16_residual_add_with_prefetch(case):
    """The BF16 add in the convolution's epilogue: several tiles per CTA, ragged tiles, channel tiles that some warps have no part
    in, sums that overflow. Both tensors equal those of the add by itself."""
    from tpu_compiler_b200 import module
    n, ic, oc, hw, mode = case
    rng = np.random.default_rng(oc)
    shape = "shape=%d,%d,%d,%d dtype=BF16" % (n, oc, hw, hw)
    text = ("input name=res %s\n" % shape + "input name=x shape=%d,%d,%d,%d dtype=BF16\n" % (n, ic, hw, hw) +
            conv_text("BF16", n, ic, oc, hw, 1, 1, 0, 1, 0) + "eltwise_add name=s in=res,c %s do_relu=1\n" % shape)
    w = {"f": graphs._bf16_np(rng.normal(0, 0.2, (oc, ic, 1, 1))), "b": rng.normal(0, 0.2, oc).astype(np.float32)}
    x = {"x": graphs._bf16_np(rng.normal(0, 1, (n, ic, hw, hw))), "res": graphs._bf16_np(rng.normal(0, 1, (n, oc, hw, hw)) * 2.0 ** rng.integers(-20, 20, (n, oc, hw, hw)))}
    x["x"][0, :, 0, 0] *= np.float32(2.0) ** 124  # sums past the largest finite value
    x["res"][0, :, 0, 0] = 3.38e38
    got = []
    for fuse in (0, mode):
        m = module(0)
        m.set_option("fuse_residual_add", fuse)
        m.load_text(text, w)
        for name, v in x.items():
            m.set_tensor(name, v)
        for _ in range(2):
            m.invoke()
        got.append([m.get_tensor(k) for k in ("c", "s")] + [m.kernel_count()])
        m.close()
    assert got[1][2] == got[0][2] - 1
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("relu", [False, True])
@pytest.mark.parametrize("shape", [(1, 1024, 96, 8, 1), (2, 144, 160, 9, 3), (1, 48, 200, 40, 5)])  # n, ic, oc, hw, k
def test_float_requantisation_past_its_range(relu, shape):
    """Sums far past the range in which the floating-point form is exact, of both signs, beside small ones: every shift for which
    the ends of the range are saturated and those just past, the smallest and largest normalised multipliers."""
    n, ic, oc, hw, k = shape
    rng = np.random.default_rng(17 + oc + relu)
    f = rng.integers(-127, 128, (oc, ic, k, k)).astype(np.float32)
    f[::3] = np.sign(f[::3]) * 127          # the largest sums
    f[1::3] = np.where(rng.random(f[1::3].shape) < 0.03, f[1::3], 0)
    past = 17 if relu else 16  # from this less one on the integer form, where sums are large
    r = (np.arange(oc) % past).astype(np.float32)
    r[oc // 2:] = rng.integers(7, 14, oc - oc // 2)
    m = (rng.integers(2 ** 23, 2 ** 24, oc) * 128).astype(np.float32)
    m[::7], m[3::7] = 2.0 ** 30, 2.0 ** 31 - 128
    b = rng.integers(-2 ** 20, 2 ** 20, oc).astype(np.float32)
    b[::11] = rng.choice([-1, 1], b[::11].shape) * np.float32(2.0) ** 27
    x = rng.integers(-128, 128, (n, ic, hw, hw)).astype(np.float32)
    x[0, :, : hw // 2] = np.sign(f[0, :, :1, :1] + 0.5) * 127  # in step with the first filter
    for top in (past, past - 1):  # with a shift that keeps the layer on the integer form, and without
        text = "input name=x shape=%d,%d,%d,%d dtype=INT8\n" % (n, ic, hw, hw) + conv_text("INT8", n, ic, oc, hw, k, 1, k // 2, 1, int(relu), True)
        got, ref = run_model(text, {"f": f, "b": b, "r": np.where(r < top, r, 9), "m": m}, {"x": x}, ["c"],
                             requant="integer" if top == past else "float")["c"]
        assert np.array_equal(got, ref)


@pytest.mark.parametrize("form", [1256, 1096, 2256, 2192, 2032])  # 1000 CTAs per tile + pixels per tile
@pytest.mark.parametrize("case", [  # n, ic, oc, hw, k, stride; shifts: the floating-point requantisation, the integer one
    (3, 64, 256, 20, 1, 1, (11, 17)), (2, 96, 136, 13, 3, 1, (11, 15)), (2, 96, 136, 13, 3, 1, (11, 17)),
    (5, 160, 300, 9, 3, 2, (11, 17)), (1, 1040, 520, 5, 1, 1, (11, 15)), (23, 80, 144, 41, 3, 1, (11, 15)), (23, 80, 144, 41, 3, 1, (11, 17))])
def test_big_tiles_with_leaky_relu(form, case):
    """Two stores per column group, the plain result and the activated one: several tiles per CTA, ragged tiles and channel tiles.
    Shifts of 15 and 16 do not saturate the ends of the floating-point form's range, which K of 720 and more weights reaches."""
    from tpu_compiler_b200 import module
    n, ic, oc, hw, k, s, shifts = case
    model = graphs.single_conv_i8(n, ic, oc, hw, k, s, k // 2, relu=False, seed=6300 + ic + k, rshift_range=shifts)
    o = (hw + 2 * (k // 2) - k) // s + 1
    text = model.text + ("leaky_relu name=lk in=conv,-,-,-,-,rp,mp,rn,mn shape=%d,%d,%d,%d dtype=INT8 negative_slope=0.1\n" % (n, oc, o, o))
    got = []
    for pos in ((4, 13), (0, 0)):  # the positive side rescaled, and as it is
        w = dict(model.weights, **{nm: np.array([v], np.float32) for nm, v in zip(("rp", "mp", "rn", "mn"), pos + (7, 12))})
        for mode in (0, form):
            m = module(0)
            m.set_option("big_tiles", mode)
            m.load_text(text, w)
            assert m.kernel_count() == 1
            requant = "integer" if shifts[1] == 17 and ic * k * k >= 720 else "float"
            assert has_form(m, "conv", tiles="big" if mode else "small", requant=requant), m.op_form("conv")
            m.set_tensor("x", model.meta["x"])
            for _ in range(2):
                m.invoke()
            got.append([m.get_tensor("conv"), m.get_tensor("lk")])
            m.close()
        if n < 23:
            ref = graph_runner.run(text, w, {"x": model.meta["x"]})
            assert all(np.array_equal(g, ref[nm]) for g, nm in zip(got[-1], ("conv", "lk")))
    assert len(np.unique(got[0][0])) > 100  # live values
    for a, b in ((0, 1), (2, 3)):
        assert np.array_equal(got[a][0], got[b][0]) and np.array_equal(got[a][1], got[b][1])


@pytest.mark.parametrize("form", [1256, 1096, 2256, 2192, 2032])
@pytest.mark.parametrize("case", [(2, 48, 144, 13, 3), (23, 16, 144, 41, 1)])  # n, ic, oc, hw, k
def test_big_tiles_write_remainders(form, case):
    """An fp32 convolution that another one reads stores its remainder operand from the same buffer, behind its result."""
    from tpu_compiler_b200 import module
    n, ic, oc, hw, k = case
    rng = np.random.default_rng(51 + oc + k)
    w = {"f": rng.normal(0, 0.1, (oc, ic, k, k)).astype(np.float32), "b": rng.normal(0, 0.2, oc).astype(np.float32),
         "g": rng.normal(0, 0.1, (64, oc, 1, 1)).astype(np.float32), "h": rng.normal(0, 0.2, 64).astype(np.float32)}
    x = rng.normal(0, 1, (n, ic, hw, hw)).astype(np.float32)
    text = ("input name=x shape=%d,%d,%d,%d dtype=FP32\n" % (n, ic, hw, hw) + conv_text("FP32", n, ic, oc, hw, k, 1, k // 2, 1, 1) +
            conv_text("FP32", n, oc, 64, hw, 1, 1, 0, 1, 0).replace("name=c in=x,f,b", "name=d in=c,g,h"))
    got = []
    for mode in (0, form):
        m = module(0)
        m.set_option("big_tiles", mode)
        m.load_text(text, w)
        assert m.kernel_count() == 3  # the pass that forms the remainder is that of x
        assert all(has_form(m, nm, tiles="big" if mode else "small") for nm in "cd")
        m.set_tensor("x", x)
        for _ in range(2):
            m.invoke()
        got.append([m.get_tensor(nm) for nm in "cd"])
        m.close()
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("scale,fused", [(0.03, True), (9.9e29, True), (-9.9e29, True), (1e30, False), (-1e30, False), (3e36, False), (3.3e38, False)])
def test_activation_chain_up_to_its_largest_scale(scale, fused):
    """The fused chain rounds its products without a check for overflow, so scales from 1e30 on keep the three ops: every byte
    value, the three tensors of the default against those of the ops by themselves."""
    from tpu_compiler_b200 import module
    base, slope = graphs.lut_slope_tables("mish")
    w = {"t0": np.tile(base, 4), "t1": np.tile(slope, 4)}
    shape = "shape=1,32,4,8"
    text = ("input name=x %s dtype=INT8\nquant name=d in=x %s dtype=BF16 from=INT8 to=BF16 scale=%r\nmish name=a in=d,t0,t1 %s dtype=BF16\n"
            "quant name=q in=a %s dtype=INT8 from=BF16 to=INT8 scale=32.0\n" % (shape, shape, scale, shape, shape))
    x = np.arange(1024, dtype=np.float32).reshape(1, 32, 4, 8) % 256 - 128
    got = []
    for on in (0, 1):
        m = module(0)
        m.set_option("fuse_activations", on)
        m.load_text(text, w)
        m.set_tensor("x", x)
        m.invoke()
        got.append([m.get_tensor(nm) for nm in "daq"] + [m.kernel_count()])
        m.close()
    assert got[0][3] == 3 and got[1][3] == (1 if fused else 3)
    assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(got[0][:3], got[1][:3]))
