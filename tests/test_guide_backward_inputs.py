"""The tensor-core backward pass's input layer at bins far from the input.

With n samples of one and the same feature vector, the gradient of W0's row k is x_k sum_t G_0[t], so
that the rows are to each other as the one-blob values x_k of their bins. Bound per row, against the
FP64 one-blob values, in the row and in the row it is compared with: a BF16 rounding (2^-9), the FP32
exponential of an argument of up to 58 with three roundings (3 * 58 * 2^-24) and the FP32 additions of
128 products (128 * 2^-24 of their absolute sum, taken as at most 10 times the sum).
"""

import numpy as np
import pytest

from oracle import guide_ref as ref


@pytest.mark.gpu
@pytest.mark.parametrize("feature", [0.0, 0.2, 0.45, 0.5, 0.53, 0.75, 1.0])
def test_input_layer_gradient_follows_the_encoding(gpu_lib, feature):
    import photon_gpu

    rng = np.random.default_rng(3)
    parts = ref.unpack(ref.init_params(4, out_scale=1.0))
    for name in ("b0", "b1", "b2", "b3", "b4"):
        parts[name] = rng.normal(0.0, 0.1, parts[name].shape)
    n = 128
    f = np.full((n, 7), feature, np.float32)
    d = np.array([0.0, 0.6, 0.8]) + 0.05 * rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    _, grads = photon_gpu.guide_gradients(ref.pack(parts), f, d, np.ones(n))
    rows = grads[:ref.IN * ref.HID].reshape(7, ref.BINS, ref.HID).astype(np.float64)
    z = float(np.float32(feature)) * ref.BINS - (np.arange(ref.BINS) + 0.5)
    x = np.exp(-0.5 * z * z)
    best = int(x.argmax())
    bound = 2 * (2.0 ** -9 + (3 * 58 + 10 * 128) * 2.0 ** -24)
    for i in range(7):
        want = rows[i, best] / x[best]
        for k in np.flatnonzero(x > 1e-25):
            err = np.linalg.norm(rows[i, k] / x[k] - want)
            assert err <= bound * np.linalg.norm(want), (i, k, x[k])
