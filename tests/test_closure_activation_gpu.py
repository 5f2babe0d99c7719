"""The closure's activation in a run (mlp_infer32) is the training pass's: on a fluid at rest the
features are (0, 0, 0, 0, 0, 0.25 log(1 + y+)), and nu_t / nu is the network of the trainer's
forward pass on them.  Both round each layer's output to BF16 and differ by the order of their
float sums only, so one BF16 rounding (2^-8) bounds the difference of the softplus."""
import numpy as np
import pytest

from cases import HW2, make_case, within

pytestmark = pytest.mark.gpu

IN, H = 6, 64


def _params(kind, rng):
    w1, b1 = np.zeros((IN, H)), np.zeros(H)
    w2, b2 = np.zeros((H, H)), np.zeros(H)
    w3, b3 = np.zeros(H), 0.0
    if kind == "tail":  # one unit far down the activation's tail, scaled back by the next layer
        b1[0], w2[0, 0], w3[0] = -50.0, 1e20, 1.0
    else:
        w1, b1 = rng.standard_normal((IN, H)), rng.standard_normal(H)
        w2, b2 = rng.standard_normal((H, H)) / 8, rng.standard_normal(H)
        w3 = rng.standard_normal(H) / 8
    return np.concatenate([w1.ravel(), b1, w2.ravel(), b2, w3, [b3]]).astype(np.float32)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["tail", "random"])
def test_run_and_training_share_the_activation(kind, precision):
    import turbchannel_b200 as tb

    prod, _, zz = make_case(HW2, 16, 16, 40, turb=1, precision=precision)
    P = _params(kind, np.random.default_rng(5))
    m = tb.Mlp(seed=1)
    m.params = P
    zc = 0.5 * (zz[1:] + zz[:-1])
    X = np.zeros((40, IN))
    X[:, 5] = 0.25 * np.log1p(np.minimum(zc - zz[0], zz[-1] - zc) * prod["inv_length_scale"])
    want = m.forward(X)
    m.close()
    S = tb.Solver(prod, zz)
    S.set_turb_model(tb.TURB_MLP, P)
    nt = np.asarray(S.RecalcTurbVisc(np.zeros((S.N, 3)))).reshape(40, -1) / prod["visc"]
    S.close()
    err = np.max(np.abs(nt - want[:, None]) / want[:, None])
    assert within(f"activation/{kind}/p{precision}", err, 2.0 ** -8), err
