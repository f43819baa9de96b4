"""Weight and bias gradients where the weight-gradient kernel marches many planes a block
(16 and 20 of the finest level's; the small volumes of the other tests march one to
three): its rings of planes come round several times and long segments meet at a seam.
Bounds as in the other gradient tests.  They show one lost halo plane: taken from the
oracle's sums on one side of a seam in the middle of 32 planes, it changes every
convolution's gradient on such data by 7% or more."""
import numpy as np
import pytest
from test_unet_grad_shapes_gpu import rel

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


@pytest.mark.parametrize("sh", [(128, 128, 32), (132, 260, 20)])
def test_gradients_of_long_columns(gpu, sh):
    from oracle import unet_ref
    from tsl_array_n_gb300.tsl_array_n import Field
    from tsl_array_n_gb300.warmstart import UNetWarmStart
    rng = np.random.default_rng(11)
    n = int(np.prod(sh))
    b = rng.standard_normal(n).astype(np.float32)
    mask = (rng.random(n) < 0.1).astype(np.uint8)
    pp = (0.01 * rng.standard_normal(n)).astype(np.float32)
    target = (0.02 * rng.standard_normal(n)).astype(np.float32)
    net = UNetWarmStart(seed=5)
    loss = net.loss_backward(sh, 1.0 / sh[0], Field("float", sh).from_array(b), Field("uint8", sh).from_array(mask),
                             Field("float", sh).from_array(pp), Field("float", sh).from_array(target))
    ref_loss, ref_g = unet_ref.loss_and_grads(net.params, b, mask, pp, target, 1.0 / sh[0], sh)
    assert abs(loss - ref_loss) <= 1e-2 * ref_loss
    g, off = net.grads, 0
    for ci, co in unet_ref.SPEC:
        nw = 27 * ci * co
        assert rel(g[off:off + nw], ref_g[off:off + nw]) < 5e-2, (ci, co)
        assert rel(g[off + nw:off + nw + co], ref_g[off + nw:off + nw + co]) < 5e-2, (ci, co, "bias")
        off += nw + co
    assert rel(g[off:], ref_g[off:]) < 5e-2
