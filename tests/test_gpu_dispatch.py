"""Dispatch rules of the tensor-core convolutions at the sizes where they change: input widths that do not fill the last
64-channel chunk, and batches on either side of the small-batch kernel's limit."""
import numpy as np
import pytest

from katago_b200 import capi
from katago_b200 import modelfile as mf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(capi.PRECISION_FP16, 0.03), (capi.PRECISION_BF16, 0.2)])
@pytest.mark.parametrize("trunk,mid", [(16, 24), (32, 48), (96, 96), (112, 40), (80, 200)])
def test_input_widths_between_chunks(prec, tol, trunk, mid, oracle):
    """Residual blocks whose widths end 8 to 56 channels into a 64-channel chunk; the chunk's other channels must count as
    zeros (they lie in the next row of the tensor).  The tolerance is the reference's reduced-precision layer tolerance
    (cpp/tests/testnn.cpp:8-15), widened for bf16's 8 mantissa bits."""
    g = mf._Gen(400 + trunk + mid)
    rng = np.random.default_rng(trunk * mid)
    mask = np.zeros((3, 19, 19), np.float32)
    mask[0] = 1; mask[1, :13, :13] = 1; mask[2, :9, :10] = 1
    layer = mf._gen_ordinary(g, trunk, mid, mf.ACT_MISH)
    x = rng.standard_normal((3, 19, 19, trunk)).astype(np.float32) * mask[..., None]
    blob = mf.layer_blob(layer)
    ref = oracle.eval_layer(blob, x, mask, trunk)
    out = capi.eval_layer(blob, x, mask, trunk, precision=prec)
    assert np.all(np.abs(out - ref) <= tol * np.maximum(np.maximum(np.abs(out), np.abs(ref)), 3.0))
