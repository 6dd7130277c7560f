"""The last-axis transforms at every length (register rows up to 512 points, line passes above) for one
row, a pair, an odd count and more rows than a CTA holds, against numpy in float64."""

import math

import numpy as np
import pytest
import torch

from oracle import spectral as S
from torchfsm_gb300 import pde

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 32, 64, 128, 256, 512, 1024, 2048, 4096])
def test_every_length_and_row_count(n):
    op = pde.Burgers(0.01)
    u = torch.randn((1, 1, n), device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    op.integrate(u_0=u, mesh=[(0.0, 1.0, n)], dt=1e-5, step=1)
    sp = op._state_dict["integrator"].spectral
    # FP32 transforms: log2(n) butterfly levels of 2^-24 each and the split, as relative rms
    tol = 6e-8 * (math.log2(n) + 2)
    for rows in (1, 2, 3, 131):
        x = torch.randn((rows, 1, n), device="cuda", generator=torch.Generator("cuda").manual_seed(rows))
        half = sp.to_half(x)
        ref = np.fft.rfft(x.cpu().numpy().astype(np.float64), axis=-1)
        assert S.rel_l2(torch.view_as_real(half).cpu().numpy(), np.stack([ref.real, ref.imag], -1)) < tol
        # the inverse of a half spectrum whose k = 0 and n/2 modes carry an imaginary part: it is dropped
        half[..., 0] += 0.5j
        half[..., -1] -= 0.25j
        back = sp.to_physical(half)
        assert S.rel_l2(back.cpu().numpy(), np.fft.irfft(half.cpu().numpy().astype(np.complex128), n=n, axis=-1)) < tol
