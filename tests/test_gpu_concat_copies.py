"""Concatenation along the channels and its split: sizes around the vector width, the unrolled trip and empty parts of a row."""
import numpy as np
import pytest

from tests.test_gpu_ops import env  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,Ca,Cb,H,W", [(1, 1, 1, 1, 1), (3, 4, 8, 1, 1), (2, 3, 5, 7, 9), (2, 64, 96, 16, 16), (1, 17, 4, 64, 64), (300, 4, 1, 2, 2), (2, 1024, 12, 4, 3)])
def test_concat_and_split(env, N, Ca, Cb, H, W):
    rng = np.random.RandomState(Ca + Cb)
    a, b = rng.randn(N, Ca, H, W).astype(np.float32), rng.randn(N, Cb, H, W).astype(np.float32)
    A, B, out = env.nd.array(a, env.ctx), env.nd.array(b, env.ctx), env.nd.empty((N, Ca + Cb, H, W), env.ctx)
    da, db = env.nd.empty(a.shape, env.ctx), env.nd.empty(b.shape, env.ctx)
    env.gpu_op.concat_forward(A, B, out, env.stream)
    env.gpu_op.concat_a_backward(A, B, out, da, env.stream)
    env.gpu_op.concat_b_backward(A, B, out, db, env.stream)
    np.testing.assert_array_equal(out.asnumpy(), np.concatenate([a, b], axis=1))
    np.testing.assert_array_equal(da.asnumpy(), a)
    np.testing.assert_array_equal(db.asnumpy(), b)
