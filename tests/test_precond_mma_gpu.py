"""The layer and weight-gradient kernels of the learned preconditioner at the edges of their
tiles: columns (site, RHS) in tiles of 8 (odd m: two sites in a lane's column pair; a last tile
that is not full), output channels in tiles of 2 and 4, input channels in steps of 2 and 4 and
chunks of 4 or 8, against the oracle; and with right-hand sides, channels, spins and single weights
of very different size, for which FP32 arithmetic needs no special case.

Tolerances: an output is a chain of at most 16 N + 1 = 65 FP32 additions per 4 input channels, so
its error is about 2^-24 sqrt(65) = 4.8e-7 of it a layer and 8.3e-7 after three layers: 2e-6 for
the output.  The gradient follows the layers and their adjoints, 1.2e-6: 4e-6."""
import numpy as np
import pytest

import qcu_mrhs_b200 as q
from qcu_mrhs_b200 import fields as F
from qcu_mrhs_b200.precond import LearnedPreconditioner, identity_weights
from tests.helpers import from_dev, rel_err, to_dev

pytestmark = pytest.mark.gpu

SHAPES = [((2, 2, 2, 2), 3, 1, 2, 1), ((4, 2, 2, 2), 2, 5, 2, 2), ((4, 2, 2, 4), 3, 3, 3, 5), ((2, 2, 4, 2), 4, 7, 2, 8),
          ((4, 4, 2, 2), 3, 8, 2, 9), ((2, 4, 2, 2), 2, 9, 3, 12), ((4, 2, 4, 2), 3, 12, 2, 13), ((6, 2, 2, 2), 4, 2, 3, 4)]


def _case(L, nc, m, layers, ch, seed, spread):
    rng = np.random.default_rng(seed)
    vh = F.half_volume(L)
    ws = [w + 0.1 * (rng.standard_normal(w.shape) + 1j * rng.standard_normal(w.shape))
          for w in identity_weights(layers, ch)]
    ws = [w.astype(np.complex64).astype(np.complex128) for w in ws]
    b = rng.standard_normal((2, vh, 4, nc, m)) + 1j * rng.standard_normal((2, vh, 4, nc, m))
    # right-hand sides of very different magnitude: each column carries its own scale
    b = (b * spread ** np.arange(m)).astype(np.complex64).astype(np.complex128)
    return F.gauge_field(L, nc, seed + 1), ws, b


@pytest.mark.parametrize("L,nc,m,layers,ch", SHAPES)
@pytest.mark.parametrize("spread", [1.0, 1e-3])
def test_apply_at_tile_edges(oracle_lib, L, nc, m, layers, ch, spread):
    g, ws, b = _case(L, nc, m, layers, ch, 100 + ch + m, spread)
    P = LearnedPreconditioner(L, nc, m, layers, ch, t_boundary=-1.0)
    P.set_weights(ws)
    P.set_gauge(to_dev(g))
    out = to_dev(np.zeros_like(b), q.SINGLE)
    P.apply(out, to_dev(b, q.SINGLE), precision=q.SINGLE)
    q.lib().qcuDeviceSynchronize()
    ref = oracle_lib.precond_apply(b, ws, g, L, -1.0)
    got = from_dev(out)
    for j in range(m):
        assert rel_err(got[..., j], ref[..., j]) <= 2e-6
    P.close()


@pytest.mark.parametrize("L,nc,m,layers,ch", SHAPES)
def test_gradient_at_tile_edges(oracle_lib, L, nc, m, layers, ch):
    kappa = 0.12
    g, ws, b = _case(L, nc, m, layers, ch, 200 + ch + m, 1.0)
    P = LearnedPreconditioner(L, nc, m, layers, ch, t_boundary=-1.0)
    P.set_weights(ws)
    P.set_gauge(to_dev(g))
    loss, grads = P.loss_grad(to_dev(b), kappa)
    ref_loss, ref_grads = oracle_lib.precond_loss_grad(b, ws, g, L, kappa, -1.0)
    assert loss == pytest.approx(ref_loss, rel=4e-6)
    for gg, rg in zip(grads, ref_grads):
        assert rel_err(gg, rg) <= 4e-6
    P.close()


def _loss_grad(L, nc, m, layers, ch, g, ws, b, kappa):
    P = LearnedPreconditioner(L, nc, m, layers, ch, t_boundary=-1.0)
    P.set_weights(ws)
    P.set_gauge(to_dev(g))
    loss, grads = P.loss_grad(to_dev(b), kappa)
    P.close()
    return loss, grads


@pytest.mark.parametrize("L,nc,m,layers,ch", [s for s in SHAPES if s[2] > 1])
@pytest.mark.parametrize("spread,period", [(1e-3, 2), (1e-6, 2), (1e-2, 4)])
def test_gradient_of_unequal_right_hand_sides(oracle_lib, L, nc, m, layers, ch, spread, period):
    """The loss divides by each right-hand side's norm: small ones have large output gradients, and
    all of them count alike in the weight gradient."""
    kappa = 0.12
    g, ws, b = _case(L, nc, m, layers, ch, 300 + ch + m, 1.0)
    b = (b * spread ** (np.arange(m) % period)).astype(np.complex64).astype(np.complex128)
    loss, grads = _loss_grad(L, nc, m, layers, ch, g, ws, b, kappa)
    ref_loss, ref_grads = oracle_lib.precond_loss_grad(b, ws, g, L, kappa, -1.0)
    assert loss == pytest.approx(ref_loss, rel=4e-6)
    for gg, rg in zip(grads, ref_grads):
        assert rel_err(gg, rg) <= 4e-6


@pytest.mark.parametrize("L,nc,m,layers,ch", SHAPES)
def test_gradient_of_unequal_spins(oracle_lib, L, nc, m, layers, ch):
    """Spin s of the input is a column of its own in the first layer's gradient: small spins to the
    tolerance of the large one."""
    kappa = 0.12
    g, ws, b = _case(L, nc, m, layers, ch, 500 + ch + m, 1.0)
    b = (b * np.array([1.0, 1e-2, 1e-3, 1e-4])[:, None, None]).astype(np.complex64).astype(np.complex128)
    _, grads = _loss_grad(L, nc, m, layers, ch, g, ws, b, kappa)
    _, ref_grads = oracle_lib.precond_loss_grad(b, ws, g, L, kappa, -1.0)
    for s in range(4):
        assert rel_err(grads[0][..., s], ref_grads[0][..., s]) <= 4e-6


@pytest.mark.parametrize("L,nc,m,layers,ch", SHAPES + [((2, 2, 2, 2), 3, 3, 1, 1)])
@pytest.mark.parametrize("octaves", [0, 10, 20])
def test_identity_network_keeps_24_bits(L, nc, m, layers, ch, octaves):
    """Entries down to 2^-21 of a column's largest pass the identity path within a unit of the last
    of 24 bits of themselves in every layer."""
    rng = np.random.default_rng(600 + ch + m)
    g, _, b = _case(L, nc, m, layers, ch, 600 + ch + m, 1.0)
    part = lambda: rng.choice([-1, 1], b.shape) * rng.uniform(0.5, 1, b.shape) * 2.0 ** -rng.uniform(0, octaves, b.shape)
    b = (part() + 1j * part()).astype(np.complex64).astype(np.complex128)
    P = LearnedPreconditioner(L, nc, m, layers, ch, t_boundary=-1.0)
    P.set_weights(identity_weights(layers, ch))
    P.set_gauge(to_dev(g))
    out = to_dev(np.zeros_like(b), q.SINGLE)
    P.apply(out, to_dev(b, q.SINGLE), precision=q.SINGLE)
    q.lib().qcuDeviceSynchronize()
    d = from_dev(out) - b
    P.close()
    assert np.all(np.abs(d.real) <= layers * 2.0 ** -23 * np.abs(b.real))
    assert np.all(np.abs(d.imag) <= layers * 2.0 ** -23 * np.abs(b.imag))


def _unequal_channels(ws, factor, balanced):
    """Channel o of every layer between two others times factor^(o mod 3), its weights in the next
    layer times the inverse (balanced: the network is the same) or as they are."""
    ws = [w.copy() for w in ws]
    for l in range(len(ws) - 1):
        d = factor ** (np.arange(ws[l].shape[0]) % 3)
        ws[l] *= d[:, None, None, None, None]
        if balanced:
            ws[l + 1] /= d[None, :, None, None, None]
    return [w.astype(np.complex64).astype(np.complex128) for w in ws]


@pytest.mark.parametrize("L,nc,m,layers,ch", [s for s in SHAPES if s[4] > 1])
@pytest.mark.parametrize("factor,balanced", [(1e-2, True), (1e-2, False), (1e-3, True)])
def test_gradient_of_unequal_channels(oracle_lib, L, nc, m, layers, ch, factor, balanced):
    """Every (output, input channel) block of the gradient to the tolerance of the whole."""
    kappa = 0.12
    g, ws, b = _case(L, nc, m, layers, ch, 400 + ch + m, 1.0)
    ws = _unequal_channels(ws, factor, balanced)
    _, grads = _loss_grad(L, nc, m, layers, ch, g, ws, b, kappa)
    _, ref_grads = oracle_lib.precond_loss_grad(b, ws, g, L, kappa, -1.0)
    for gg, rg in zip(grads, ref_grads):
        for o in range(rg.shape[0]):
            for i in range(rg.shape[1]):
                assert rel_err(gg[o, i], rg[o, i]) <= 4e-6


def _apply(L, nc, m, layers, ch, g, ws, b):
    P = LearnedPreconditioner(L, nc, m, layers, ch, t_boundary=-1.0)
    P.set_weights(ws)
    P.set_gauge(to_dev(g))
    out = to_dev(np.zeros_like(b), q.SINGLE)
    P.apply(out, to_dev(b, q.SINGLE), precision=q.SINGLE)
    q.lib().qcuDeviceSynchronize()
    P.close()
    return from_dev(out)


@pytest.mark.parametrize("L,nc,m,layers,ch", [s for s in SHAPES if s[4] > 1])
@pytest.mark.parametrize("factor", [1e-2, 1e-5, 1e-9])
def test_apply_with_unequal_channels(oracle_lib, L, nc, m, layers, ch, factor):
    """Factors shifted between a channel and its weights leave the network and its errors alone."""
    g, ws, b = _case(L, nc, m, layers, ch, 700 + ch + m, 1.0)
    ws = _unequal_channels(ws, factor, True)
    ref = oracle_lib.precond_apply(b, ws, g, L, -1.0)
    assert rel_err(_apply(L, nc, m, layers, ch, g, ws, b), ref) <= 2e-6


@pytest.mark.parametrize("L,nc,m,layers,ch", [s for s in SHAPES if s[4] > 1])
def test_apply_of_a_small_row(oracle_lib, L, nc, m, layers, ch):
    """An output channel of tiny weights beside ordinary ones, and nothing else of the layer in the
    output."""
    g, ws, b = _case(L, nc, m, layers, ch, 800 + ch + m, 1.0)
    ws[0][1] *= 1e-10
    ws[1][:, [i for i in range(ch) if i != 1]] = 0.0
    ws = [w.astype(np.complex64).astype(np.complex128) for w in ws]
    ref = oracle_lib.precond_apply(b, ws, g, L, -1.0)
    assert rel_err(_apply(L, nc, m, layers, ch, g, ws, b), ref) <= 2e-6


@pytest.mark.parametrize("L,nc,m,layers,ch", SHAPES)
@pytest.mark.parametrize("size", [1e34, 1e-30])
def test_apply_keeps_the_range_of_fp32(oracle_lib, L, nc, m, layers, ch, size):
    g, ws, b = _case(L, nc, m, layers, ch, 900 + ch + m, 1.0)
    b = (b * size).astype(np.complex64).astype(np.complex128)
    ref = oracle_lib.precond_apply(b, ws, g, L, -1.0)
    assert rel_err(_apply(L, nc, m, layers, ch, g, ws, b), ref) <= 2e-6


# more columns than one wave of the MMA kernel's tiles: FP32 arithmetic in the layers that it suits
# (one channel on a side, few channels, SU(2) and SU(4) with 6), the MMA in the others and where a
# block would not hold m channels threads
LARGE = [((8, 8, 4, 6), 3, 7, 3, 2), ((8, 6, 6, 6), 2, 6, 3, 6), ((6, 8, 6, 6), 4, 6, 3, 6), ((8, 8, 8, 4), 3, 5, 3, 5),
         ((8, 4, 6, 8), 3, 9, 3, 3), ((4, 4, 4, 4), 3, 64, 2, 8), ((6, 6, 6, 8), 4, 6, 1, 1)]


@pytest.mark.parametrize("L,nc,m,layers,ch", LARGE)
def test_layers_of_large_lattices(oracle_lib, L, nc, m, layers, ch):
    kappa = 0.12
    g, ws, b = _case(L, nc, m, layers, ch, 1100 + ch + m, 1.0)
    ref = oracle_lib.precond_apply(b, ws, g, L, -1.0)
    assert rel_err(_apply(L, nc, m, layers, ch, g, ws, b), ref) <= 2e-6
    loss, grads = _loss_grad(L, nc, m, layers, ch, g, ws, b, kappa)
    ref_loss, ref_grads = oracle_lib.precond_loss_grad(b, ws, g, L, kappa, -1.0)
    assert loss == pytest.approx(ref_loss, rel=4e-6)
    for gg, rg in zip(grads, ref_grads):
        assert rel_err(gg, rg) <= 4e-6


def test_gradient_beside_an_infinite_channel(oracle_lib):
    """A channel whose output gradient overflows (its last weight is near FP32's largest number, its
    own value is zero) leaves the other channels' gradients as they are."""
    L, nc, m, ch, kappa = (4, 2, 2, 4), 3, 8, 4, 0.12
    g, ws, b = _case(L, nc, m, 2, ch, 1000, 1.0)
    ws[0][2] = 0.0
    ws[1][0, 2] = 0.0
    ws[1][0, 2, 0] = 3e38 * np.eye(4)
    ws = [w.astype(np.complex64).astype(np.complex128) for w in ws]
    _, grads = _loss_grad(L, nc, m, 2, ch, g, ws, b * 1e-5, kappa)
    _, ref = oracle_lib.precond_loss_grad(b * 0.01, ws, g, L, kappa, -1.0)
    assert not np.all(np.isfinite(grads[0][2]))
    for o in (0, 1, 3):
        assert rel_err(grads[0][o], ref[0][o]) <= 4e-6
        assert rel_err(grads[1][0, o], ref[1][0, o]) <= 4e-6
