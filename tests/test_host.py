"""CPU-side checks: the C-ABI library loads and exports every symbol include/tpucb.h declares,
fails loudly without a GPU, and the host-side graph builders agree with the oracle."""
import ctypes as C
import os
import re

import numpy as np
import pytest

import oracle
from oracle import graph_runner
from tpu_compiler_b200 import _lib, graphs

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "tpucb.h")).read()
    return sorted(set(re.findall(r"\b(tpucb_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    L = _lib.lib()
    names = _declared_symbols()
    assert len(names) >= 25
    for n in names:
        assert hasattr(L, n), n
    assert L.tpucb_version() >= 1


def test_no_gpu_fails_loudly():
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    L = _lib.lib()
    h = C.c_void_p()
    assert L.tpucb_interp_create(0, C.byref(h)) != 0
    msg = L.tpucb_last_error().decode()
    assert "no CPU fallback" in msg


def test_numpy_requant_matches_oracle():
    rng = np.random.default_rng(3)
    v = rng.integers(-2 ** 31, 2 ** 31, 5000)
    m = (rng.integers(2 ** 30, 2 ** 31 - 128, 5000) // 128) * 128
    r = rng.integers(0, 32, 5000)
    got = graphs.qdm_np(v, m, r)
    L = oracle.lib()
    exp = np.array([L.orc_qdm_i32(int(a), int(c), int(b)) for a, b, c in zip(v, m, r)])
    assert np.array_equal(got, exp)


def test_quantize_multiplier_range():
    for q in (0.9, 0.5, 0.123, 1e-3, 3e-6):
        m, r = graphs.quantize_multiplier(q)
        assert 2 ** 30 <= m < 2 ** 31 and 0 <= r <= 31
        assert float(np.float32(m)) == m
        assert abs(m / 2 ** 31 / 2 ** r - q) / q < 1e-6


def test_builder_simulation_matches_oracle_graph():
    """The scale-picking simulation inside the builder and the oracle agree on a small
    residual network, tensor by tensor (bit-exact INT8)."""
    b = graphs.GraphBuilder(11, simulate=True)
    img = np.random.default_rng(5).uniform(-1, 1, (1, 3, 20, 20))
    b.input("data", (1, 3, 20, 20), sample=img)
    x = b.quant_in("q", "data", 1.0)
    x = b.conv_i8("c1", x, 32, 3, stride=2, pad=1)
    x = b.pool_max("p1", x, 3, 2, pad=(0, 1, 0, 1))
    y = b.conv_i8("c2", x, 16, 1, pad=0)
    y = b.conv_i8("c3", y, 16, 3, pad=1)
    y = b.conv_i8("c4", y, 32, 1, pad=0, relu=False)
    x = b.eltwise_add_i8("add", [x, y])
    x = b.pool_avg_i8("gap", x)
    x = b.fc_i8("fc", x, 10)
    T = graph_runner.run(b.text(), b.weights, {"data": img.astype(np.float32)})
    for name in ("q", "c1", "p1", "c2", "c3", "c4", "add", "gap", "fc"):
        assert np.array_equal(T[name].reshape(-1), b.sim[name].astype(np.float32).reshape(-1)), name
    assert T["c3"].std() > 5  # the synthetic scales keep a live dynamic range


def test_resnet50_graph_shape():
    m = graphs.resnet50_int8(batch=1, simulate=False)
    ops = graph_runner.parse(m.text)
    assert sum(o["type"] == "conv_2d" for o in ops) == 53
    assert sum(o["type"] == "eltwise_add" for o in ops) == 16
    macs = 0
    for o in ops:
        if o["type"] == "conv_2d":
            w = m.weights[o["in"][1]]
            macs += int(np.prod(o["shape"])) * int(np.prod(w.shape[1:]))
    assert 3.8e9 < macs < 4.2e9


def _build_worker(args):
    """One process of test_concurrent_builds: points the build module at a scratch library and a fake compiler."""
    lib_path, log_path = args
    import subprocess
    import time
    from tpu_compiler_b200 import build as b
    b.LIB = lib_path

    def fake_compiler(cmd, check=True):
        out = cmd[cmd.index("-o") + 1]
        assert out != lib_path, "the compiler must not write the library in place"
        with open(out, "wb") as f:
            f.write(b"half")
            f.flush()
            time.sleep(0.3)   # a reader that opened the final path now would see a truncated file
            f.write(b"-written-library")
        with open(log_path, "a") as f:
            f.write("compiled\n")
        return subprocess.CompletedProcess(cmd, 0)

    b.build(run=fake_compiler)
    with open(lib_path, "rb") as f:
        return f.read()


def test_concurrent_builds(tmp_path):
    """Two ranks that both find the library stale: one compiles (into a temporary file, renamed over the library),
    the other waits on the lock, sees a fresh library and does not compile; neither reads a partial file."""
    import multiprocessing as mp
    lib_path, log_path = str(tmp_path / "libfake.so"), str(tmp_path / "log.txt")
    with mp.get_context("spawn").Pool(2) as pool:
        got = pool.map(_build_worker, [(lib_path, log_path)] * 2)
    assert got == [b"half-written-library"] * 2
    assert open(log_path).read().count("compiled") == 1
    assert [f for f in os.listdir(tmp_path) if f.endswith(".tmp")] == []


COPY_HELPERS = r"""
#include "host_copy.h"
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <dlfcn.h>
#include <pthread.h>
#include <sys/wait.h>
#include <vector>

static std::atomic<int> may_start{1 << 30}; // threads that may still be created
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *x) {
  if (may_start.fetch_sub(1) <= 0) return EAGAIN;
  static auto real = (int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *))dlsym(RTLD_NEXT, "pthread_create");
  return real(t, a, f, x);
}

static bool copies(unsigned seed, int rounds) {
  const size_t block = 64u << 10;
  std::vector<uint8_t> src(37 * block + 4321);
  uint8_t *dst = (uint8_t *)aligned_alloc(64, 38 * block);
  bool good = true;
  for (int r = 0; r < rounds; ++r) {
    const int n = 1 + (r * 7 + seed) % 38;
    const size_t len = n == 38 ? src.size() : n * block;
    for (size_t i = 0; i < len; i += 97) src[i] = (uint8_t)(i * 31 + r + seed);
    std::atomic<int> done{0};
    int calls = 0;
    tpucb::CopyHelpers::run(
        n, true,
        [&](int i) {
          tpucb::stream_copy(dst + i * block, src.data() + i * block, std::min(block, len - i * block));
          done.fetch_add(1);
        },
        [&] { ++calls; return done.load() == n; });
    good = good && calls >= 1 && done.load() == n && std::memcmp(dst, src.data(), len) == 0;
  }
  free(dst);
  return good;
}

int main(int argc, char **argv) {
  if (argc > 1) may_start = atoi(argv[1]);
  if (!copies(0, 50)) return 1;
  if (argc > 1) return 0;
  std::atomic<int> bad{0};
  std::vector<std::thread> users;
  for (unsigned t = 1; t <= 4; ++t) users.emplace_back([&, t] { if (!copies(t, 200)) ++bad; });
  for (auto &u : users) u.join();
  const pid_t child = fork();
  if (child == 0) _exit(copies(9, 50) ? 0 : 1); // the helpers of the parent are not there
  int status = 1;
  waitpid(child, &status, 0);
  return bad || status || !copies(10, 50);
}
"""


def test_copy_helpers_threads_fork_and_thread_limit(tmp_path):
    """The copies of set_tensor on several host threads: four threads at once, a forked child, and a process that may start
    no helper, one or two."""
    import subprocess
    src, exe = tmp_path / "t.cpp", str(tmp_path / "t")
    src.write_text("#include <algorithm>\n#include <cstdint>\n" + COPY_HELPERS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "tpu_compiler_b200", "csrc"), str(src), "-o", exe,
                    "-ldl"], check=True)
    for args in ([], ["0"], ["1"], ["2"]):
        assert subprocess.run([exe] + args, timeout=120).returncode == 0, args


KERNELS_READY = r"""
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <map>
#include <mutex>
#include <thread>
static thread_local int current_device = 0;
static std::mutex m;
static std::map<std::pair<int, const void *>, int> set_up;
static int failing = 0; // calls that report an error yet
static cudaError_t fake_get_device(int *d) { *d = current_device; return cudaSuccess; }
template <class Kernel> cudaError_t fake_set_attribute(Kernel k, cudaFuncAttribute, int) {
  std::lock_guard<std::mutex> g(m);
  if (failing > 0 && failing--) return cudaErrorInvalidValue;
  ++set_up[{current_device, (const void *)k}];
  return cudaSuccess;
}
#define cudaGetDevice fake_get_device
#define cudaFuncSetAttribute fake_set_attribute
#include "conv_plan.cuh"

int main() {
  tpucb::ConvPlan i8, tf32;
  std::memset(&i8.p, 0, sizeof(i8.p));
  i8.p.fastq = 1;
  std::memset(&tf32.p, 0, sizeof(tf32.p));
  tf32.tf32 = true;
  for (int device : {0, 1, 0, 1}) { // as a module on the first device and then one on the second would
    current_device = device;
    tpucb::conv_kernel_ready(i8);
    tpucb::conv_kernel_ready(tf32);
  }
  if (set_up.size() != 4) return 1;
  current_device = 2;
  failing = 1;
  try { // an error of the driver leaves the device to the next caller
    tpucb::conv_kernel_ready(i8);
    return 2;
  } catch (const tpucb::Error &) {
  }
  tpucb::conv_kernel_ready(i8);
  std::vector<std::thread> users;
  for (int t = 0; t < 8; ++t)
    users.emplace_back([&] {
      current_device = 3;
      tpucb::conv_kernel_ready(i8);
    });
  for (auto &u : users) u.join();
  for (auto &k : set_up)
    if (k.second != 1) return 3;
  return set_up.size() == 6 ? 0 : 4;
}
"""


def test_kernels_are_set_up_on_every_device(tmp_path):
    """A kernel's limit of shared memory belongs to a device: what plans call at load sets it once on each (the driver's calls
    are replaced here), again after an error, and once for several threads."""
    import subprocess
    from tpu_compiler_b200 import build as b
    src, exe = tmp_path / "t.cu", str(tmp_path / "t")
    src.write_text(KERNELS_READY)
    subprocess.run([b._nvcc(), "-gencode", "arch=compute_100a,code=compute_100a", "-std=c++17", "-O0", "-I", b.CSRC, str(src), "-o", exe], check=True)
    assert subprocess.run([exe], timeout=120).returncode == 0


RESIDUAL_ADDS = r"""
#include "module_text.h"
#include <iostream>
int main(int argc, char **argv) {
  std::vector<tpucb::ParsedOp> ops;
  std::map<std::string, const tpucb::ParsedOp *> by_name;
  std::map<std::string, int> n_uses;
  for (std::string line; std::getline(std::cin, line);) ops.push_back(tpucb::parse_line(line));
  for (auto &op : ops) {
    by_name[op.name] = &op;
    for (auto &nm : op.in) n_uses[nm]++;
  }
  for (auto &name : tpucb::residual_add_tails(ops, by_name, n_uses, atoi(argv[1]), atoi(argv[2]))) std::cout << name << std::endl;
}
"""


@pytest.fixture(scope="module")
def add_tails(tmp_path_factory):
    import subprocess
    from tpu_compiler_b200 import build as b
    d = tmp_path_factory.mktemp("add_tails")
    (d / "t.cu").write_text(RESIDUAL_ADDS)
    subprocess.run([b._nvcc(), "-gencode", "arch=compute_100a,code=compute_100a", "-std=c++17", "-I", b.CSRC, str(d / "t.cu"), "-o", str(d / "t")], check=True)

    def run(text, fuse=2, batch=1):
        return subprocess.run([str(d / "t"), str(fuse), str(batch)], input=text, text=True, check=True, capture_output=True).stdout.split()
    return run


def _residual(dtype="BF16", n=32, ic=64, oc=256, hw=28, conv="", add="do_relu=1", add_in="r,c", extra="", res="input"):
    s = "shape=%d,%%d,%d,%d dtype=%s" % (n, hw, hw, dtype)
    tail = ",-,-,ar,am" if dtype == "INT8" else ""
    return ("input name=x " + s % ic + "\n%s name=r%s " % (res, "" if res == "input" else " in=x") + s % oc + "\nconv_2d name=c in=x,f,b " + s % oc +
            " kh=1 kw=1 sh=1 sw=1 %s\neltwise_add name=s in=%s%s " % (conv, add_in, tail) + s % oc + " %s\n%s" % (add, extra))


@pytest.mark.parametrize("case,kept", [
    (dict(), True), (dict(add_in="c,r"), True), (dict(add="do_relu=1 coeff=1.0,1"), True),
    (dict(add="do_relu=0"), False), (dict(add="do_relu=1 coeff=1.0,0.5"), False),   # the epilogue's BF16 add has a ReLU and no coefficients
    (dict(conv="do_relu=1"), False), (dict(conv="g=2"), False), (dict(add_in="c,c"), False), (dict(add_in="r,c,x"), False),
    (dict(extra="relu name=q in=c shape=32,256,28,28 dtype=BF16\n"), False),      # a second reader of the convolution
    (dict(res="reshape"), False), (dict(add_in="r,w"), False),
    (dict(n=1, hw=50), False), (dict(n=2, hw=51), True),                           # 1.22 and 2.54 MiB
    (dict(ic=256, n=10, hw=28), True), (dict(ic=256, n=11, hw=28), False)])        # 3.83 and 4.21 MiB of a layer that does not widen
def test_layers_give_up_large_tiles_only_for_an_add_they_take(add_tails, case, kept):
    assert add_tails(_residual(**case)) == (["c"] if kept else [])


def test_layers_that_give_up_large_tiles_by_option(add_tails):
    assert add_tails(_residual(), fuse=0) == []
    assert add_tails(_residual(n=1, hw=50), fuse=1) == ["c"]            # every add
    assert add_tails(_residual(n=1, hw=50), fuse=2, batch=3) == ["c"]   # the size is that of all batch slots
    assert add_tails(_residual("INT8"), fuse=1) == ["c"]
    assert add_tails(_residual("INT8", n=100, ic=1536, oc=2048), fuse=2) == ["c"]                 # 12 K blocks, 153 MiB
    k3 = "kh=3 kw=3 pt=1 pb=1 pl=1 pr=1"
    assert add_tails(_residual("INT8", n=26, ic=256, oc=512, conv=k3), fuse=2) == ["c"]           # 18 blocks, 9.95 MiB
    assert add_tails(_residual("INT8", n=27, ic=256, oc=512, conv=k3), fuse=2) == []              # 10.3 MiB: the loop counts, not the add
    assert add_tails(_residual("INT8", n=10, ic=257, oc=512, conv=k3), fuse=2) == []              # 27
    assert add_tails(_residual("INT8", n=27, ic=257, oc=512, conv=k3), fuse=1) == ["c"]
    assert add_tails(_residual("FP32"), fuse=1) == []
