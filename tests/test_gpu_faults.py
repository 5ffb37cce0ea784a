"""Error paths, exercised without faulting, trapping or hanging anything: a bounded device wait that runs out (a
barrier that nothing arrives at; no copy in flight) comes back as an error status and leaves the interpreter usable;
malformed modules are refused at load with a status."""
import numpy as np
import pytest

from oracle import graph_runner
from tpu_compiler_b200 import graphs

pytestmark = pytest.mark.gpu


def test_bounded_wait_runs_out_and_the_interpreter_stays_usable():
    from tpu_compiler_b200 import TpucbError, module
    # 784 pixel tiles on 296 persistent CTAs: some CTAs own three tiles, and the third needs an accumulator buffer
    # back from the epilogue. With the self-test option the epilogue never hands it back.
    model = graphs.single_conv_i8(64, 64, 64, 56, 3, 1, 1, seed=31)
    m = module(0)
    m.set_option("selftest_lost_arrival", 4)       # every wait: 4 rounds of 1024 polls
    m.load_text(model.text, model.weights)
    m.set_tensor("x", model.meta["x"])
    with pytest.raises(TpucbError, match="bounded wait"):
        m.invoke()
    with pytest.raises(TpucbError, match="bounded wait"):
        m.invoke()                                  # the same module fails the same way again: nothing is left wedged
    # the same interpreter, the same module without the self-test: correct results
    m.set_option("selftest_lost_arrival", 0)
    m.load_text(model.text, model.weights)
    m.set_tensor("x", model.meta["x"])
    m.invoke()
    ref = graph_runner.run(model.text, model.weights, {"x": model.meta["x"]})["conv"]
    assert np.array_equal(m.get_tensor("conv"), ref)
    m.close()
    # and a fresh interpreter on the same device works too (the context survived)
    small = graphs.single_conv_i8(1, 32, 32, 8, 3, 1, 1, seed=5)
    s = module(0)
    s.load_text(small.text, small.weights)
    out = s.run(small.meta["x"])["conv"]
    assert np.array_equal(out, graph_runner.run(small.text, small.weights, {"x": small.meta["x"]})["conv"])
    s.close()


def test_malformed_modules_are_refused_with_a_status():
    from tpu_compiler_b200 import TpucbError, module
    model = graphs.single_conv_i8(1, 32, 32, 8, 3, 1, 1, seed=6)
    m = module(0)
    # a filter of the wrong size
    w = dict(model.weights)
    w["conv_filter"] = w["conv_filter"][:, :, :, :2]
    with pytest.raises(TpucbError, match="filter has"):
        m.load_text(model.text, w)
    # a multiplier outside [0, 2^31): the reference's quantiser emits none, the epilogue could not represent it
    w = dict(model.weights)
    mult = w["conv_multiplier"].copy()
    mult[3] = np.float32(2 ** 31)
    w["conv_multiplier"] = mult
    with pytest.raises(TpucbError, match="outside"):
        m.load_text(model.text, w)
    w["conv_multiplier"] = -model.weights["conv_multiplier"]
    with pytest.raises(TpucbError, match="outside"):
        m.load_text(model.text, w)
    # an operand that does not exist, an INT8 convolution without its requantisation operands
    with pytest.raises(TpucbError):
        m.load_text(model.text.replace("in=x,", "in=y,"), model.weights)
    with pytest.raises(TpucbError, match="rshift and multiplier"):
        m.load_text(model.text.replace("conv_rshift,conv_multiplier", "-,-"), model.weights)
    # after all that the interpreter still loads and runs the good module
    m.load_text(model.text, model.weights)
    out = m.run(model.meta["x"])["conv"]
    assert np.array_equal(out, graph_runner.run(model.text, model.weights, {"x": model.meta["x"]})["conv"])
    m.close()


@pytest.mark.parametrize("form,dtype", [
    ("big_tiles 1256", "INT8"), ("big_tiles 2256", "INT8"), ("fused add", "INT8"), ("small tiles", "BF16"), ("big_tiles 1256", "BF16"),
    ("big_tiles 2256", "BF16"), ("fused add", "BF16"), ("small tiles", "FP32"), ("big_tiles 1256", "FP32"), ("big_tiles 2256", "FP32"),
    ("stem", "FP32")])
def test_bounded_wait_runs_out_in_the_other_forms(form, dtype):
    """The kernels whose epilogue warps meet at barriers, and the image stem: after the MMA issuer's wait and then theirs have run
    out, every warp (and both CTAs of a pair) still leaves, and the interpreter stays usable."""
    from tpu_compiler_b200 import TpucbError, module
    n, ic, oc = (16, 3, 64) if form == "stem" else (64, 64, 256)
    k, hw = (1, 56) if form == "fused add" else ((3, 56) if form == "stem" else (3, 28))  # more than two tiles per CTA
    if dtype == "INT8":
        model = graphs.single_conv_i8(n, ic, oc, hw, k, 1, k // 2, relu=False, seed=37)
        text, w, x = model.text, dict(model.weights), {"x": model.meta["x"]}
    else:
        rng = np.random.default_rng(37)
        cut = graphs._bf16_np if dtype == "BF16" else (lambda v: np.asarray(v, np.float32))
        w = {"f": cut(rng.normal(0, 0.1, (oc, ic, k, k))), "b": rng.normal(0, 0.2, oc).astype(np.float32)}
        x = {"x": cut(rng.normal(0, 1, (n, ic, hw, hw)))}
        text = ("input name=x shape=%d,%d,%d,%d dtype=%s\nconv_2d name=conv in=x,f,b shape=%d,%d,%d,%d dtype=%s kh=%d kw=%d sh=1 sw=1 pt=%d "
                "pb=%d pl=%d pr=%d dh=1 dw=1 g=1 do_relu=0 with_bias=1\n" % ((n, ic, hw, hw, dtype, n, oc, hw, hw, dtype, k, k) + (k // 2,) * 4))
    names = ["conv"]
    if form == "fused add":
        shape = "shape=64,256,%d,%d dtype=%s" % (hw, hw, dtype)
        text = "input name=res %s\n" % shape + text + "eltwise_add name=s in=res,conv%s %s do_relu=1\n" % (",-,-,ar,am" if dtype == "INT8" else "", shape)
        w.update(ar=np.array([7.0], np.float32), am=np.array([70.0, 60.0], np.float32))
        x["res"], names = np.random.default_rng(3).integers(-128, 128, (64, 256, hw, hw)).astype(np.float32), ["conv", "s"]
    got = []
    m = module(0)
    for rounds in (4, 0):
        m.set_option("selftest_lost_arrival", rounds)
        if form == "fused add":
            m.set_option("fuse_residual_add", 1 if rounds else 0)
        else:
            m.set_option("big_tiles", int(form.split()[1]) if rounds and form.startswith("big") else 0)
        m.load_text(text, w)
        if rounds:
            assert m.op_form("conv")["tiles"] == {"big": "big", "ste": "stem"}.get(form[:3], "small")
            assert m.kernel_count() == (2 if dtype == "FP32" and form != "stem" else 1)  # fp32: the pass that forms the remainder
        for name, v in x.items():
            m.set_tensor(name, v)
        if rounds:
            for _ in range(2):
                with pytest.raises(TpucbError, match="bounded wait"):
                    m.invoke()
        else:
            m.invoke()
            got.append([m.get_tensor(n) for n in names])
    m.set_option("fuse_residual_add", 1)
    m.set_option("big_tiles", int(form.split()[1]) if form.startswith("big") else 1)
    m.load_text(text, w)
    for name, v in x.items():
        m.set_tensor(name, v)
    m.invoke()
    assert all(np.array_equal(a, m.get_tensor(n)) for a, n in zip(got[0], names))
    m.close()
