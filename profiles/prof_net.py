"""One eager launch of a module between cudaProfilerStart and cudaProfilerStop, for ncu --profile-from-start off.

    python profiles/prof_net.py <graph of tpu_compiler_b200.graphs> <batch>
    python profiles/prof_net.py conv <batch> <c_in> <c_out> <hw> <k> <relu>
    python profiles/prof_net.py conv_add <batch> <c_in> <c_out> <hw>   (a 1x1 layer and the INT8 residual add behind it)
    python profiles/prof_net.py calibration <batch>          (two batches of the fp32 ResNet-50)
"""
import os
import re
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import numpy as np
import torch

from tpu_compiler_b200 import graphs, module
from tpu_compiler_b200.calibration import ActivationCalibrator


def profiled(work):
    torch.cuda.cudart().cudaProfilerStart()
    work()
    torch.cuda.cudart().cudaProfilerStop()


kind, batch = sys.argv[1], int(sys.argv[2])
if kind == "conv":
    c_in, c_out, hw, k, relu = (int(v) for v in sys.argv[3:8])
    model = graphs.single_conv_i8(1, c_in, c_out, hw, k, 1, k // 2, relu=bool(relu))
elif kind == "conv_add":
    c_in, c_out, hw = (int(v) for v in sys.argv[3:6])
    model = graphs.single_conv_i8(1, c_in, c_out, hw, 1, 1, 0, relu=False)
    shape = "shape=1,%d,%d,%d dtype=INT8" % (c_out, hw, hw)
    model.text = "%sinput name=res %s\neltwise_add name=sum in=res,conv,-,-,ar,am %s do_relu=1\n" % (model.text, shape, shape)
    lines = model.text.splitlines()
    model.text = "\n".join([lines[-2]] + lines[:-2] + [lines[-1]]) + "\n"  # the residual is there before the convolution
    model.weights.update(ar=np.array([7.0], np.float32), am=np.array([70.0, 60.0], np.float32))
elif kind == "calibration":
    model = graphs.resnet50_fp32(1)
else:
    model = getattr(graphs, kind)(1, **({"simulate": False} if kind.startswith("yolo") else {}))
m = module(0)
m.load_text(re.sub(r"shape=1\b", "shape=%d" % batch, model.text), model.weights)
if kind == "calibration":
    data = [torch.randn(batch, 3, 224, 224).clamp_(-3, 3).pin_memory() for _ in range(2)]
    cal = ActivationCalibrator(m, lambda: iter(data))
    cal.run()
    profiled(cal.run)
else:
    m.set_option("cuda_graph", 0)
    name = "x" if kind == "conv_add" else m.get_input_details()[0]
    x = np.random.default_rng(0).uniform(-1, 1, m.get_tensor_shape(name)).astype(np.float32)
    m.set_tensor(name, np.rint(x * 127) if kind.startswith("conv") else x)
    m.launch()
    m.launch()
    m.sync()
    profiled(lambda: (m.launch(), m.sync()))
print("done", kind, batch, m.kernel_count())
