"""The device-pointer products (qt_mode_product, qt_hole_product) at the edges
of their kernels' tiles: hole products split over thread groups and clusters
of CTAs (tile sides 15..17, one output, rectangular, up to the largest
accepted number of columns, reductions shorter than a staged chunk and not a
multiple of the CTA count), mode products of one output per thread.  Bound:
every output is a sum of K complex products whose partial sums are added in
some order, so |err| <= 4 (K + 8) 2^-53 sum |a| |b| (four real products and
sums per complex multiply-add)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def ctx():
    from qutree_gb300.qtgpu import Context
    c = Context(0)
    yield c
    c.close()


def _rand(rng, *shape):
    return np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))


@pytest.mark.parametrize("before,aA,aB,after", [
    (1, 1, 1, 1), (1, 1, 1, 5000), (5000, 1, 1, 1), (63, 6, 6, 1), (33, 15, 17, 1), (1, 16, 16, 31),
    (1, 17, 33, 32), (29, 16, 16, 11), (7, 3, 50, 37), (1, 400, 400, 3), (2, 90, 110, 65), (257, 31, 16, 2),
    (8, 64, 64, 8), (4096, 2, 2, 3)])
def test_hole_product_edges(ctx, before, aA, aB, after):
    rng = np.random.default_rng(before + 3 * aA + 5 * aB + 7 * after)
    A, B = _rand(rng, before, aA, after), _rand(rng, before, aB, after)
    ref = np.einsum("bic,bjc->ij", A.conj(), B, optimize=True)
    bound = np.einsum("bic,bjc->ij", abs(A), abs(B), optimize=True)
    dA, dB = ctx.to_device(A.ravel(order="F")), ctx.to_device(B.ravel(order="F"))
    dS = ctx.to_device(np.full(aA * aB, np.nan, complex))
    ctx.hole_product(dS, dA, dB, before, aA, aB, after)
    got = ctx.from_device(dS, (aA * aB,)).reshape((aA, aB), order="F")
    for p in (dA, dB, dS):
        ctx.free(p)
    assert (abs(got - ref) <= 4 * (before * after + 8) * EPS * bound).all()


@pytest.mark.parametrize("before,aB,aC,after", [(1, 1, 1, 1), (1, 7, 5, 3), (31, 4, 6, 9), (257, 3, 1, 1), (1, 130, 2, 129)])
@pytest.mark.parametrize("add", [False, True])
def test_mode_product_edges(ctx, before, aB, aC, after, add):
    rng = np.random.default_rng(before + 3 * aB + 5 * aC + 7 * after)
    B, h, C0 = _rand(rng, before, aB, after), _rand(rng, aC, aB), _rand(rng, before, aC, after)
    ref = np.einsum("ja,bac->bjc", h, B) + (C0 if add else 0)
    bound = np.einsum("ja,bac->bjc", abs(h), abs(B)) + (abs(C0) if add else 0)
    dB, dh, dC = (ctx.to_device(x.ravel(order="F")) for x in (B, h, C0))
    ctx.mode_product(dC, dh, dB, before, aB, aC, after, add=add)
    got = ctx.from_device(dC, (C0.size,)).reshape(C0.shape, order="F")
    for p in (dB, dh, dC):
        ctx.free(p)
    assert (abs(got - ref) <= 4 * (aB + 8) * EPS * bound).all()
