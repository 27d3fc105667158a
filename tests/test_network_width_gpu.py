"""The network built in other shapes (-DDG_NN_WIDTH, -DDG_NN_DEPTH).  128 wide its training pass does not fit
one kernel and runs as the chain of one kernel per product (k_gemm, k_loss), which no other test reaches; the
other shapes train in one kernel (k_train) with other operand sizes, column counts and numbers of links.  A
library with that network code is linked here (the step's kernels in it keep the default shape: only the
network's own calls are made) and a child process runs the network's tests on it."""
import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = pathlib.Path(__file__).resolve().parent


def library(out, width, depth):
    from dumses_hybrid_b200 import build
    objs = [build.BUILD / (s + ".o") for s in [*build.CU_SOURCES, *build.CXX_SOURCES] if s != "nn_flux.cu"]
    if not all(o.exists() for o in objs):
        build.build(force=True)
    obj, lib = out / "nn_flux.o", out / "libdumses_gpu_shape.so"
    build._run([build._nvcc(), *build.NVCC_FLAGS, *build.CU_SOURCES["nn_flux.cu"], f"-DDG_NN_WIDTH={width}", f"-DDG_NN_DEPTH={depth}",
                "-c", str(build.CSRC / "nn_flux.cu"), "-o", str(obj)], False)
    build._run([build._nvcc(), *build.ARCH, "-shared", "-cudart", "static", "-Xcompiler", "-fPIC", *map(str, objs),
                str(obj), "-o", str(lib)], False)
    return lib


def child(lib, *args):
    res = subprocess.run([sys.executable, *args], capture_output=True, text=True, timeout=600, cwd=str(HERE.parent),
                         env=dict(os.environ, DG_LIBRARY=str(lib)))
    assert res.returncode == 0, res.stdout[-3000:] + res.stderr[-3000:]
    return res.stdout


ORACLE = ["tests/test_nn_gpu.py::" + n for n in ("test_forward_matches_oracle", "test_gradients_match_oracle",
                                                 "test_adam_step_matches_oracle")] + ["tests/test_train_tiles_gpu.py"]


def run_tests(lib, *tests):
    out = child(lib, "-m", "pytest", "-q", "-p", "no:cacheprovider", *tests)
    assert " passed" in out and "skipped" not in out, out


@pytest.mark.parametrize("width,depth", [(32, 2), (64, 1), (64, 3)])
def test_one_kernel_shapes(tmp_path, built_library, width, depth):
    run_tests(library(tmp_path, width, depth), *ORACLE, "tests/test_train_sums_gpu.py", "tests/test_train_wait_gpu.py")


def sums():
    """Weight gradients of a batch: the in-order sum of its 512-row pieces' gradients, bit for bit (the bias
    sums of the chain add their four warps in any order); the same after a larger batch of fewer splits."""
    from test_nn_gpu import FluxNet, layer_slices, random_params
    rng = np.random.default_rng(7)
    x = rng.normal(0, 1, (65536, 17)).astype(np.float32)
    t = rng.normal(0, 1, (65536, 8)).astype(np.float32)
    few = 128 * 299  # 299 splits of 128 rows
    with FluxNet() as net:
        assert net.shape[0] == 128
        random_params(net, 12)
        weights = layer_slices(net)[::2]
        alone = net.gradients(x[:few], t[:few])[1]
    with FluxNet() as net:
        random_params(net, 12)
        net.gradients(x, t)  # 128 splits of 512 rows
        again = net.gradients(x[:few], t[:few])[1]
        got = net.gradients(x[:4096], t[:4096])[1]
        want = np.zeros(net.param_count, np.float32)
        for a in range(0, 4096, 512):
            want += net.gradients(x[a:a + 512], t[a:a + 512])[1] * np.float32(1 / 8)
    for s in weights:
        assert np.array_equal(again[s], alone[s]) and np.array_equal(got[s], want[s])
    print("sums held")


def test_kernel_chain(tmp_path, built_library):
    lib = library(tmp_path, 128, 2)
    run_tests(lib, *ORACLE)
    assert "sums held" in child(lib, "-c", f"import sys; sys.path[:0] = ['.', {str(HERE)!r}]; "
                                "import test_network_width_gpu as t; t.sums()")
