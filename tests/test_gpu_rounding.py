"""Rounding error that a flow gathers without reunitarisation (FP64 flows have
none): lattices that run one launch per stage stay as close to the flow in higher
precision as the stage kernels of larger ones, whose links see the same local
arithmetic whatever the volume."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS, EPS, A = 400, 0.01, 0.35


def rms(links, want):
    return np.sqrt(((links - want) ** 2).sum() / (want.size // 2))  # per complex entry


def fp32_error(n, precision):
    from latticeyangmills_b200 import GluonField

    out = []
    for p in ("fp64", precision):
        with GluonField(n, p) as f:
            f.init_links("expiah", A, 1)
            f.flow(EPS, STEPS, 0)
            out.append(f.download())
    return rms(out[1], out[0])


@pytest.mark.parametrize("precision", ["fp32_18", "fp32_12"])
def test_fp32_small_lattices_drift_no_faster_than_large_ones(precision):
    # 8^4 (16,384 links) and 8^3 x 10 differ by a few per cent from seed to seed
    small, large = fp32_error((8, 8, 8, 8), precision), fp32_error((8, 8, 8, 10), precision)
    print(precision, "rms |dU| after", STEPS, "steps:", small, "against", large)
    assert small < 1.15 * large


def extended_flow(U, n):
    """The flow of U in extended precision, from the definitions (staples,
    Luscher's third-order Runge-Kutta, e^{iQ} by its power series)."""
    real = np.longdouble
    a = U.reshape(n[3], n[2], n[1], n[0], 4, 3, 3, 2).astype(real)
    u = [np.moveaxis(a[..., m, :, :, 0] + 1j * a[..., m, :, :, 1], (4, 5), (0, 1)) for m in range(4)]
    one = np.eye(3, dtype=u[0].dtype).reshape(3, 3, 1, 1, 1, 1)

    def mul(x, y):
        return x[:, 0:1] * y[0:1] + x[:, 1:2] * y[1:2] + x[:, 2:3] * y[2:3]

    def dag(x):
        return x.transpose(1, 0, 2, 3, 4, 5).conj()

    def shift(x, mu, sign):
        return np.roll(x, -sign, axis=5 - mu)

    def force(mu):
        omega = 0
        for nu in range(4):
            if nu != mu:
                up = shift(u[nu], mu, 1)
                omega = omega + mul(mul(up, dag(shift(u[mu], nu, 1))), dag(u[nu]))
                omega = omega + shift(mul(mul(dag(up), dag(u[mu])), u[nu]), nu, -1)
        x = mul(u[mu], omega)
        z = real(0.5) * 1j * (x - dag(x))
        return z - one * (z[0, 0] + z[1, 1] + z[2, 2]) / real(3)

    def exp_i(q):
        x = 1j * q
        e = one + x / real(14)
        for k in range(13, 0, -1):
            e = one + mul(x, e) / real(k)
        return e

    eps, z = real(EPS), [0] * 4
    for _ in range(STEPS):
        for new, old, e in ((real(1), real(0), eps / 4), (real(8) / 9, -real(17) / 36, eps), (real(3) / 4, -real(1), eps)):
            z = [new * force(mu) + old * z[mu] for mu in range(4)]
            u = [mul(exp_i(e * z[mu]), u[mu]) for mu in range(4)]
    m = np.stack([np.moveaxis(x, (0, 1), (4, 5)) for x in u], 4)
    return np.stack([m.real, m.imag], -1).reshape(U.shape)


def test_fp64_small_lattices_drift_no_faster_than_large_ones(oracle):
    """Against extended precision.  The two-kernel stage of larger lattices
    gathers 7.6e-16 per entry over these steps (8^3 x 10: about
    sqrt(1200 stages) roundings of 2e-17), whatever the volume."""
    from latticeyangmills_b200 import GluonField

    n = (4, 4, 4, 4)
    U = oracle.gen_expiah(n, A, 1, 0)
    with GluonField(n, "fp64") as f:
        f.upload(U)
        f.flow(EPS, STEPS, 0)
        links = f.download()
    err = float(rms(links, extended_flow(U, n)))
    print("rms |dU| after", STEPS, "steps:", err)
    assert err < 1.15 * 7.6e-16
