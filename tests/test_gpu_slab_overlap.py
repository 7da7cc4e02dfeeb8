"""Slab transform of one rank whose send buffer lies over the real slab (the planes' spectrum then
goes through the handle's own buffer)."""
import ctypes as C

import numpy as np
import pytest

from meumapps_ss_b200 import _lib
from meumapps_ss_b200 import params as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [P.PREC_F64, P.PREC_F32])
@pytest.mark.parametrize("shift", [0, 1024, -1024])
def test_send_buffer_over_the_real_slab(prec, shift):
    import torch
    L = _lib.lib()
    nx, ny, nz = 32, 24, 18
    rd = torch.float64 if prec == P.PREC_F64 else torch.float32
    x = np.random.default_rng(4).standard_normal((nz, ny, nx))
    spec = np.fft.rfftn(x) / x.size
    h = C.c_void_p()
    assert L.meu_slab_fft_create(nx, ny, nz, 1, 0, prec, C.byref(h)) == 0
    need = 2 * nz * ny * (nx // 2 + 1)
    pool = torch.zeros(need + 4096, dtype=rd, device="cuda")
    real = pool[1024:1024 + nx * ny * nz]
    send = pool[1024 + shift:1024 + shift + need]
    real.copy_(torch.tensor(x, dtype=rd).reshape(-1))
    assert L.meu_slab_fft_forward_planes(h, C.c_void_p(real.data_ptr()), C.c_void_p(send.data_ptr()), None) == 0
    assert L.meu_slab_fft_forward_columns(h, C.c_void_p(send.data_ptr()), None) == 0
    torch.cuda.synchronize()
    got = send.cpu().numpy().astype(np.float64).view(np.complex128).reshape(nz, ny, nx // 2 + 1)
    # FP64: the gate of the transforms' own tests; FP32 likewise
    assert np.max(np.abs(got - spec)) <= (1e-12 if prec == P.PREC_F64 else 3e-6) * np.max(np.abs(spec))
    assert L.meu_slab_fft_destroy(h) == 0
