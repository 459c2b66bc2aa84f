"""Networks with xnor layers: the order in which their dense layers add is the reference's, and the same at every batch size.

The layers after them take signs, so the last bit of a sum can decide a whole +1 or -1."""
import hashlib

import numpy as np
import pytest

import darknet_b200 as dn
from darknet_b200 import synth

pytestmark = pytest.mark.gpu


def network(cfg, params, tmp_path, mode=dn.MODE_TF32):
    path = str(tmp_path / "n.weights")
    synth.write_weights(path, params)
    return dn.Network(cfg, path, mode, text=True)


def octet_cases(size):
    """(a, b) of the products a, b that end a full group of eight of the im2col order, and lie at different taps."""
    taps = size * size
    for g in range(3 * taps // 8):
        for a, b in ((8 * g, 8 * g + 7), (8 * g + 1, 8 * g + 6)):
            if a % taps != b % taps:
                yield a, b


@pytest.mark.parametrize("size,stride", [(3, 1), (3, 2), (5, 1), (7, 2)])
def test_first_layer_adds_in_the_im2col_order(size, stride, tmp_path):
    """All inputs are 1.  Filter f has +2^30 and -2^30 at two products of one group of eight and 1 at every product after that
    group: added in the im2col order, eight at a time, the large ones cancel before the first small one comes, and the sum is the
    number of small ones, exactly.  In any order that adds a small one between them it is lost (2^30 + 1 is not a float)."""
    k_all = 3 * size * size
    pairs = list(octet_cases(size))[:32]
    n = (len(pairs) + 15) // 16 * 16
    cfg = synth._net(2, 40, 24) + synth._conv(n, size, stride=stride, bn=False, act="linear") + synth._conv(32, 3, xnor=True)
    params = synth.seeded_params(cfg, 1)
    w, want = np.zeros((n, k_all), np.float32), np.zeros(n, np.float32)
    for f, (a, b) in enumerate(pairs):
        after = 8 * (b // 8) + 8
        w[f, a], w[f, b], w[f, after:] = 2.0 ** 30, -2.0 ** 30, 1.0
        want[f] = k_all - after
    params[0].weights[...] = w.reshape(params[0].weights.shape)
    params[0].biases[...] = 0
    net = network(cfg, params, tmp_path)
    assert net.layer_kernel(0) == "stem_tc_tf32"
    net.predict(np.ones((2, 3, 24, 40), np.float32))
    inner = net.layer_output(0).reshape((2,) + net.layer_shape(0))[:, :, 4:-4, 4:-4]     # whole receptive fields
    assert np.array_equal(inner, np.broadcast_to(want[None, :, None, None], inner.shape))
    net.close()


def digest(a):
    return hashlib.sha256(np.ascontiguousarray(a, np.float32).tobytes()).hexdigest()[:16]


def test_binarised_darknet19_is_pinned(tmp_path):
    """Darknet-19 with xnor layers at 224, batch 128: first-layer values and the network's answers, to the bit (recorded with the first
    layer in the im2col order on the tensor cores), and an image's answer does not depend on the batch it came in."""
    cfg = synth.darknet19_cfg(batch=128, size=224, xnor=True)
    params, x = synth.seeded_params(cfg, 21), synth.seeded_input(cfg, 22)
    net = network(cfg, params, tmp_path)
    want = net.predict(x).reshape(128, -1).copy()
    first = net.layer_output_images(0, 40, 4)
    net.close()
    assert (digest(first), digest(want)) == ("1d314ae047462e3f", "3a52b9dfc6aef328")
    for batch in (1, 6):
        small = network(synth.darknet19_cfg(batch=batch, size=224, xnor=True), params, tmp_path)
        for at in (0, 122):
            assert np.array_equal(small.predict(x[at:at + batch]).reshape(batch, -1), want[at:at + batch])
        small.close()


@pytest.mark.parametrize("mode,groups", [(dn.MODE_FP32, 1), (dn.MODE_FP32, 2), (dn.MODE_TF32, 2)])
@pytest.mark.parametrize("batch", [1, 26])     # small and large tiles of the fp32 GEMM
def test_dense_layers_on_cuda_cores_add_in_the_reference_order(mode, groups, batch, tmp_path):
    """A 3x3 layer between others, channels-last: inputs are 1, +2^30 and -2^30 lie at the first and the last tap of a group's
    first channel, 1 at every product after them.  In the order c, kh, kw the sum is the number of small ones, exactly."""
    cpg, npg = 24 // groups, 40 // groups
    cfg = (synth._net(batch, 40, 40) + synth._conv(24, 3, bn=False, act="linear") + synth._conv(40, 3, bn=False, act="linear", groups=groups) +
           synth._conv(32, 3, xnor=True))
    params = synth.seeded_params(cfg, 1)
    params[0].weights[...], params[0].biases[...] = 0, 1
    w = np.ones((40, cpg * 9), np.float32)
    w[:, 0], w[:, 1:8], w[:, 8] = 2.0 ** 30, 0, -2.0 ** 30
    params[1].weights[...], params[1].biases[...] = w.reshape(params[1].weights.shape), 0
    net = network(cfg, params, tmp_path, mode)
    assert net.layer_kernel(1) == "direct_fp32" and npg > 16
    net.predict(np.zeros((batch, 3, 40, 40), np.float32))
    inner = net.layer_output(1).reshape((batch,) + net.layer_shape(1))[:, :, 1:-1, 1:-1]
    assert (inner == 9 * (cpg - 1)).all()
    net.close()


def test_shortcuts_of_another_shape_keep_their_roundings(tmp_path):
    """In front of an xnor layer: the convolution's output is rounded to TF32, the sum with an addend of fewer channels and twice the
    map is not, as the two layers do it one by one.  Computed here from the two layers' own outputs, to the bit."""
    cfg = (synth._net(3, 20, 20, 16) + synth._conv(64, 3) + synth._conv(96, 3, stride=2, act="linear") + synth._shortcut(-2, "leaky") +
           synth._conv(32, 3, xnor=True))
    net = network(cfg, synth.seeded_params(cfg, 4), tmp_path)
    net.predict(synth.seeded_input(cfg, 5, "normal"))
    out = [net.layer_output(i).reshape((3,) + net.layer_shape(i)) for i in range(3)]
    want = out[1].copy()
    want[:, :64] += out[0][:, :, ::2, ::2]
    want = np.where(want > 0, want, np.float32(0.1) * want)
    assert np.array_equal(out[2], want)
    net.close()
