"""Schedules of the one-CTA tensor-core kernel: shared activation blocks, resident filters, clusters, accumulator layouts."""
import numpy as np
import pytest

from tests.test_gpu_ops import env  # noqa: F401

pytestmark = pytest.mark.gpu


# N, C, H, W, K, R, S, padding
@pytest.mark.parametrize("case", [
    (16, 64, 5, 5, 64, 3, 3, "SAME"),         # all nine taps in one block
    (2, 64, 9, 29, 96, 3, 3, "SAME"),         # two rows of taps in a block
    (1, 72, 6, 61, 132, 3, 3, "SAME"),        # one row of taps in a block, ragged channels
    (3, 128, 30, 7, 64, 7, 1, "SAME"), (3, 64, 7, 30, 200, 1, 7, "SAME"),
    (12, 64, 42, 42, 64, 3, 3, "SAME"),       # more tiles than SMs: filters stay in shared memory
    (13, 64, 40, 40, 256, 1, 1, "VALID"), (13, 248, 40, 41, 60, 1, 1, "VALID"),
    (2, 384, 8, 8, 384, 1, 3, "SAME"), (9, 1024, 4, 4, 96, 1, 1, "SAME"), (2, 512, 6, 6, 136, 3, 3, "SAME"), (5, 256, 17, 17, 160, 3, 3, "SAME"),    # few tiles: clusters of several sizes
    (9, 36, 9, 9, 44, 5, 5, "SAME"), (9, 33 * 4, 9, 9, 68, 1, 7, "SAME"), (4, 160, 12, 12, 64, 7, 1, "SAME"), (4, 320, 9, 9, 136, 1, 3, "SAME"),        # filters: more taps than a block holds, ragged blocks; gradients: taps of 3 and 5 half tiles
    (20, 512, 30, 30, 128, 3, 3, "SAME"),     # cross terms promoted twice in a tile
])
@pytest.mark.parametrize("arith", ["3xfp16", "3xtf32"])
def test_convolution_schedules(env, case, arith):
    N, C, H, W, K, R, S, padding = case
    rng = np.random.RandomState(C + K + W)
    x, w = rng.randn(N, C, H, W).astype(np.float32), rng.randn(K, C, R, S).astype(np.float32)
    out, cell = env.gpu_op.convolution_2d_forward_get_out_shape(x.shape, w.shape, "NCHW", padding, 1, 1)
    dy = rng.randn(*out).astype(np.float32)

    def run(path, x, w, dy):
        X, Wd, DY = (env.nd.array(v, env.ctx) for v in (x, w, dy))
        y, dx, dw = env.nd.empty(out, env.ctx), env.nd.empty(x.shape, env.ctx), env.nd.empty(w.shape, env.ctx)
        env.gpu_op.set_contraction_path(path)
        env.gpu_op.set_tensor_arithmetic(arith)
        try:
            env.gpu_op.convolution_2d_forward(X, Wd, y, cell, env.cudnn, env.stream)
            env.gpu_op.convolution_backward_data(X, DY, Wd, dx, cell, env.cudnn, env.stream)
            env.gpu_op.convolution_backward_filter(X, DY, Wd, dw, cell, env.cudnn, env.stream)
        finally:
            env.gpu_op.set_contraction_path(0)
            env.gpu_op.set_tensor_arithmetic("3xfp16")
        return [v.asnumpy().astype(np.float64) for v in (y, dx, dw)]

    got, want, mag = run(2, x, w, dy), run(1, x, w, dy), run(1, np.abs(x), np.abs(w), np.abs(dy))
    for name, g, e, m in zip(("forward", "backward-data", "backward-filter"), got, want, mag):
        assert np.all(np.abs(g - e) <= 2e-6 * m + 1e-30), (name, float(np.max(np.abs(g - e) / (m + 1e-30))))


@pytest.mark.parametrize("case", [
    (64, 256, 29, 29, 512, 3, 3, "SAME"),     # 72 tiles in 2 ranges, two sums each: running sums end after 384 stages
    (7, 192, 24, 24, 64, 1, 1, "VALID"),      # 2 tiles of 63 stages in 31 ranges
    (3, 100, 31, 17, 140, 3, 3, "SAME"),      # 18 tiles in 8 ranges, ragged everywhere
])
@pytest.mark.parametrize("arith", ["3xfp16", "3xtf32"])
def test_reductions_cut_at_common_stages(env, case, arith):
    test_convolution_schedules(env, case, arith)


# K, C, R, S: enough blocks that a block takes 9 taps, or 288 channels of a 1x1 filter
@pytest.mark.parametrize("filters", [[(1024, 1160, 1, 1), (640, 1000, 1, 1), (256, 268, 3, 3), (100, 300, 1, 7), (36, 32, 5, 5)], [(512, 512, 3, 3), (260, 100, 1, 1)]])
@pytest.mark.parametrize("arith", ["3xfp16", "3xtf32"])
def test_filters_packed_in_one_launch(env, filters, arith):
    rng = np.random.RandomState(len(filters))
    calls = []
    env.gpu_op.set_tensor_arithmetic(arith)
    try:
        for K, C, R, S in filters:
            x, w = rng.randn(2, C, 21, 21).astype(np.float32), rng.randn(K, C, R, S).astype(np.float32)
            out, cell = env.gpu_op.convolution_2d_forward_get_out_shape(x.shape, w.shape, "NCHW", "SAME", 1, 1)
            calls.append([env.nd.array(v, env.ctx) for v in (x, w, rng.randn(*out).astype(np.float32), np.zeros(w.shape, np.float32))] + [cell])

        def run(path):
            env.gpu_op.set_contraction_path(path)
            results = []
            for x, w, dy, _, cell in calls:
                y, dx = env.nd.empty(dy.shape, env.ctx), env.nd.empty(x.shape, env.ctx)
                env.gpu_op.convolution_2d_forward(x, w, y, cell, env.cudnn, env.stream)
                env.gpu_op.convolution_backward_data(x, dy, w, dx, cell, env.cudnn, env.stream)
                results.append((y.asnumpy(), dx.asnumpy()))
            env.gpu_op.set_contraction_path(0)
            return results
        want = run(2)                            # each filter packed on its own
        for x, w, dy, zero, cell in calls:
            env.gpu_op.sgd_update(w, zero, 1.0, env.stream)        # a new version of the same values, and its maximum
        env.gpu_op.pack_filters([c[1] for c in calls], env.gpu_op.cell_array([c[4] for c in calls]), env.stream)
        got, exact = run(2), run(1)
        for shape, g, w, e in zip(filters, got, want, exact):
            for a, b, c in zip(g, w, e):
                np.testing.assert_array_equal(a, b, err_msg=str(shape))
                np.testing.assert_allclose(a, c, rtol=1e-4, atol=2e-5 * np.abs(c).max(), err_msg=str(shape))
    finally:
        env.gpu_op.set_contraction_path(0)
        env.gpu_op.set_tensor_arithmetic("3xfp16")


# N, C, H, W, K, R, S, padding, stride: rows in one block and in several, windows past the edges, columns that are no multiple of 8
@pytest.mark.parametrize("case", [(2, 15, 9, 90, 16, 7, 7, "SAME", 1), (5, 3, 33, 47, 64, 3, 3, "SAME", 1), (2, 3, 75, 75, 64, 7, 7, "VALID", 2), (1, 3, 41, 1201, 32, 7, 7, "SAME", 3),
                                  (9, 1, 40, 41, 32, 5, 5, "SAME", 1), (9, 12, 64, 64, 64, 1, 1, "VALID", 1)])
@pytest.mark.parametrize("arith", ["3xfp16", "3xtf32"])
def test_first_layers_as_patches(env, case, arith):
    N, C, H, W, K, R, S, padding, u = case
    rng = np.random.RandomState(C + W)
    x, w = rng.randn(N, C, H, W).astype(np.float32), rng.randn(K, C, R, S).astype(np.float32)
    out, cell = env.gpu_op.convolution_2d_forward_get_out_shape(x.shape, w.shape, "NCHW", padding, u, u)
    dy = rng.randn(*out).astype(np.float32)

    def run(path, x, w, dy):
        X, Wd, DY = (env.nd.array(v, env.ctx) for v in (x, w, dy))
        y, dw = env.nd.empty(out, env.ctx), env.nd.empty(w.shape, env.ctx)
        env.gpu_op.set_contraction_path(path)
        env.gpu_op.set_tensor_arithmetic(arith)
        try:
            env.gpu_op.convolution_2d_forward(X, Wd, y, cell, env.cudnn, env.stream)
            env.gpu_op.convolution_backward_filter(X, DY, Wd, dw, cell, env.cudnn, env.stream)
        finally:
            env.gpu_op.set_contraction_path(0)
            env.gpu_op.set_tensor_arithmetic("3xfp16")
        return [v.asnumpy().astype(np.float64) for v in (y, dw)]

    for g, e, m in zip(run(2, x, w, dy), run(1, x, w, dy), run(1, np.abs(x), np.abs(w), np.abs(dy))):
        assert np.all(np.abs(g - e) <= 2e-6 * m + 1e-30), float(np.max(np.abs(g - e) / (m + 1e-30)))


@pytest.mark.parametrize("case", [(8, 64, 32, 32, 128, 1, 1, "VALID"), (33, 64, 16, 16, 192, 1, 1, "VALID"),       # 64 and 66 wide tiles
                                  (2, 2048, 8, 8, 132, 1, 1, "VALID"), (2, 2112, 8, 8, 132, 1, 1, "VALID"), (2, 224, 9, 9, 100, 3, 3, "SAME")])      # 32, 33 and 36 stages
@pytest.mark.parametrize("arith", ["3xfp16", "3xtf32"])
def test_narrow_tiles_of_short_reductions(env, case, arith):
    test_convolution_schedules(env, case, arith)


# the first product of a process asks how many clusters fit on the device before it launches anything
_FIRST_PRODUCT = """
import ctypes, json
import numpy as np
from tinyflow_b200 import gpu_op, ndarray as nd
from tinyflow_b200._base import _LIB
ctx, stream = nd.gpu(0), gpu_op.create_cudaStream()
handle = gpu_op.create_cudnnHandle(stream)
gpu_op.set_tensor_arithmetic("%s")
shape, filters = (2, 768, 17, 17), (192, 768, 1, 1)
out, cell = gpu_op.convolution_2d_forward_get_out_shape(shape, filters, "NCHW", "SAME", 1, 1)
x, w, y = (nd.array(np.ones(s, np.float32), ctx) for s in (shape, filters, out))
for step in range(2):
    _LIB.TfKernelTimingEnable(1)
    gpu_op.convolution_2d_forward(x, w, y, cell, handle, stream)
    gpu_op.device_synchronize()
    report = ctypes.create_string_buffer(1 << 16)
    _LIB.TfKernelTimingReport(report, len(report))
    print([r["name"] for r in json.loads(report.value.decode())])
"""


@pytest.mark.parametrize("arith", ["3xfp16", "3xtf32"])
def test_a_first_product_is_cut_over_clusters(lib_path, arith):
    import os
    import re
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    ran = subprocess.run([sys.executable, "-c", _FIRST_PRODUCT % arith], cwd=root, env=dict(os.environ, TINYFLOW_TIMING_DETAIL="1"), capture_output=True, text=True, timeout=300)
    lines = ran.stdout.strip().splitlines()
    assert ran.returncode == 0 and len(lines) == 2 and lines[0] == lines[1], ran.stdout + ran.stderr
    assert int(re.search(r" cl(\d+) ", lines[0]).group(1)) > 1, lines[0]
