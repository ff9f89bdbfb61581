"""Power spectra summed by groups of lanes: row lengths around the group sizes
(8 and 32 lanes, two values per lane and step), batches that end within a warp
and coefficients that are only 8-byte aligned, against the oracle's serial sums.
Sums of n positive terms, each side off by at most n rounding errors of 2^-53 of
the sum: |difference| <= 2 (n + 3) 2^-53 of it, n = 2 (l + 1) values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def device(c):
    import torch
    t = torch.zeros(c.size + 1, dtype=torch.float64, device="cuda")[1:]  # 8 bytes off a 16-byte boundary
    t.copy_(torch.from_numpy(np.ascontiguousarray(c).ravel()))
    return t


@pytest.mark.parametrize("L", [1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 48, 65, 130, 257])
def test_spectra(oracle, L):
    import zest_gb300 as zg
    ctx = zg.Context(0)
    rng = np.random.default_rng(L)
    batch = 3
    a = rng.normal(size=(batch, zg.st_coeff_size(L), 2))
    l = np.repeat(np.arange(L), np.arange(1, L + 1))
    a[:, l * (l + 1) // 2, 1] = 0.0
    got = ctx.st_power_spectrum(device(a), L, batch=batch).cpu().numpy().reshape(batch, L)
    bound = 2.0 * (2.0 * np.arange(1, L + 1) + 3.0) * 2.0 ** -53
    for b in range(batch):
        want = oracle.st_power_spectrum(a[b], L, 0)
        assert np.all(np.abs(got[b] - want) <= bound * want)
    if L > 130:
        return
    c = rng.normal(size=(batch, zg.zt_coeff_size(L), 2))
    size = ((L + 1) * (L + 1)) // 4
    z = ctx.zt_power_spectrum(device(c), L, batch=batch).cpu().numpy().reshape(batch, size)
    for b in range(batch):
        want = oracle.zt_power_spectrum(c[b], L, 0, out=np.zeros(size))
        assert np.all(np.abs(z[b] - want) <= 2.0 * (2.0 * L + 3.0) * 2.0 ** -53 * want)
    ctx.close()
