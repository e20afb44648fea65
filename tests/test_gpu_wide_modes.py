"""Mode indices beyond 32 bits: a field of N = 92684 has more than 2^32 modes a component."""

import pytest
import torch

import azeban_b200 as az  # noqa: F401
from azeban_b200 import _lib

pytestmark = pytest.mark.gpu


def test_energy_of_a_mode_beyond_32_bits():
    """One mode off k = 0, whose index is 2^32, counts twice (it stands for its conjugate too); cut to 32
    bits the index is that of mode 0, which counts once.  Scaled to energy 1 the mode is N^2."""
    N = 92684
    nh = N // 2 + 1
    if torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("needs 69 GB")
    assert 2 ** 32 < N * nh and 2 ** 32 % nh not in (0, nh - 1)
    u = torch.zeros((2, N, nh), dtype=torch.complex64, device="cuda")
    try:
        flat = u.view(-1)
        flat[2 ** 32] = 1.0
        _lib.check(_lib.lib.az_init_normalize_energy(2, N, 1, u.data_ptr(), 1, 1.0, None))
        torch.cuda.synchronize()
        assert abs(flat[2 ** 32].item()) == pytest.approx(float(N) ** 2, rel=1e-6)
    finally:
        del u, flat
        torch.cuda.empty_cache()
