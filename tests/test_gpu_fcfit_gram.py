"""
tvbg_fcfit_loss at the edges of its tiles: 4 x 4, 2 x 4 and 1 x 4 pairs a thread
(chosen by the number of instances and nodes), ragged rows and columns, the
last pass of fewer than 32 samples, and the sample and node tiles of dL/dX.

Against torch FP64 autograd of the same loss, with the bounds of the kernel's
arithmetic: the Gram's 4e-12 worst case is 1e-14 in practice (FC 1e-12, loss
1e-10), dL/dX is FP32 (1e-5).
"""

import ctypes

import pytest

from conftest import rel_err
from test_gpu_adjoint import fc_loss_torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('I,T,N', [(100, 70, 85), (45, 33, 83), (1, 31, 2), (3, 32, 3), (9, 65, 31),
                                   (1300, 34, 18), (2, 127, 32), (1, 128, 33), (2, 129, 64), (1, 257, 65),
                                   (2, 64, 96), (1, 65, 97), (2, 63, 128), (1, 64, 129)])
def test_fcfit_loss_tiles(cuda, I, T, N):
    from tvb_hpc import _native as nat
    torch = cuda
    lib = nat.load()
    g = torch.Generator(device='cuda').manual_seed(I + T + N)
    # lane-interleaved groups of 8; the idle lanes of the last one stay unread
    G = -(-I // 8)
    x = torch.rand(G, T, N, 8, device='cuda', generator=g) + 0.1
    X = x.permute(0, 3, 1, 2).reshape(G * 8, T, N)[:I]
    target = torch.corrcoef(torch.rand(N, 40, device='cuda', generator=g).double())
    loss_ref, fc_ref, dx_ref = fc_loss_torch(X, target)
    nb = ctypes.c_int64()
    nat.check(lib.tvbg_fcfit_scratch_bytes(I, N, ctypes.byref(nb)))
    scratch = torch.empty(nb.value, dtype=torch.uint8, device='cuda')
    loss = torch.empty(I, dtype=torch.float64, device='cuda')
    fc = torch.empty(I, N, N, dtype=torch.float64, device='cuda')
    dx = torch.full((I, T + 1, N), 7.0, device='cuda')
    nat.check(lib.tvbg_fcfit_loss(x.data_ptr(), T * N * 8, None, 0, 0, 8, I, T, N, target.data_ptr(),
                                  loss.data_ptr(), dx.data_ptr(), (T + 1) * N, fc.data_ptr(),
                                  scratch.data_ptr(), None))
    torch.cuda.synchronize()
    assert rel_err(fc.cpu().numpy(), fc_ref.cpu().numpy()) < 1e-12
    assert rel_err(loss.cpu().numpy(), loss_ref.cpu().numpy()) < 1e-10
    assert rel_err(dx[:, :T].cpu().numpy(), dx_ref.cpu().numpy()) < 1e-5
    assert bool((dx[:, T] == 7.0).all())
