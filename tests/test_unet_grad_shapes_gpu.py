"""Weight and bias gradients of the warm-start network at volumes that are not
whole 8 x 16 tiles, down to one voxel on the coarsest level, against the PyTorch
FP32 oracle.  Both round to BF16 at the same places and differ in the FP32
order of the sums, so a parameter block agrees within 5e-2 relative L2, the
bound of the other gradient tests (a value next to a rounding boundary may round
the other way, 2^-8 of it, and the layers below carry that on)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("sh", [(8, 4, 4), (20, 12, 4), (36, 20, 12), (68, 8, 40), (16, 16, 64)])
def test_gradients_at_ragged_volumes(gpu, sh):
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
