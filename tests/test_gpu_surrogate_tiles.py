"""The surrogate's fused gradient at one tile of rows, two, and more tiles
than thread blocks, against the CPU restatement with the same BF16 rounding."""
import numpy as np
import pytest

from md_engine_b200 import systems
from oracle import surrogate_ref as SR

pytestmark = pytest.mark.gpu


def _surrogate(rows):
    sysd = systems.water_tip4p2005(nside=6, seed=5)
    st, fx = systems.build_water_state(sysd, rcut=6.5, skin=1.0, grid=32, e3b=True)
    st.prepare()
    rng = np.random.default_rng(rows)
    w = np.zeros(SR.N_PARAMS, np.float32)
    for k, (o, s) in SR.OFF.items():
        fan = SR.N_IN if k == "W1" else SR.N_HID
        w[o:o + s] = rng.uniform(-1, 1, s) * (np.sqrt(6.0 / fan) if k.startswith("W") else 0.1)
    e3 = fx["e3b"]
    e3.surrogateSetParams(w, np.zeros(SR.N_IN), np.ones(SR.N_IN), 1.0)
    x = rng.standard_normal((rows, SR.N_IN)).astype(np.float32)
    t = rng.standard_normal((rows, SR.N_OUT)).astype(np.float32)
    return st, e3, w, x, t


@pytest.mark.parametrize("rows", [64, 128, 64 * 301])
def test_gradient_by_tiles(rows):
    st, e3, w, x, t = _surrogate(rows)
    loss, g = e3.surrogateGrad(x, t)
    lr, gr = SR.mlp_loss_grad(w, x, t)
    assert loss == pytest.approx(lr, rel=1e-2)
    # the rounding points are the same; values whose FP32 and FP64 sums round
    # to different BF16 neighbours (2^-8 apart) leave well under 2 % of the norm
    for k, (o, s) in SR.OFF.items():
        rk = np.linalg.norm(g[o:o + s] - gr[o:o + s]) / np.linalg.norm(gr[o:o + s])
        assert rk < 2e-2, (k, rk)


# three and seven tiles, a tile to each of 64 blocks, two and three to each of 148
@pytest.mark.parametrize("rows", [192, 448, 4096, 64 * 301])
def test_gradient_repeats_bit_for_bit(rows):
    st, e3, _, x, t = _surrogate(rows)
    loss, g = e3.surrogateGrad(x, t)
    for _ in range(5):
        loss2, g2 = e3.surrogateGrad(x, t)
        assert loss2 == loss and np.array_equal(g2, g)
