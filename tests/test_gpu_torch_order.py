"""A call whose inputs are still being computed on torch's current stream reads their
final values: it equals, bit for bit, the call made after torch.cuda.synchronize().  The
producer waits behind a kernel of some tens of milliseconds, far longer than a call's
host preparation."""
import numpy as np
import pytest

from test_gpu_utr import as_msk
from utr_cases import params

pytestmark = pytest.mark.gpu

CYCLES = 100_000_000  # of the delaying kernel


def late(torch, values):
    """A tensor that takes `values` only behind the delaying kernel."""
    t = torch.zeros_like(values)
    torch.cuda.synchronize()
    torch.cuda._sleep(CYCLES)
    t.copy_(values)
    return t


@pytest.mark.parametrize("side_stream", [False, True])
def test_adjoint(ctx, msk, side_stream):
    torch = pytest.importorskip("torch")
    g = torch.Generator().manual_seed(1)
    v = (torch.rand((2, 4, 64, 64), generator=g) * 40.0).cuda()
    target = (1.0 + 0.1 * torch.rand((2, 1, 64, 64), generator=g)).cuda()
    st = msk.Stack()
    st.nx = st.ny = 64
    st.ax = st.by = 20.0
    st.v0, st.deltaz, st.nslices = 200.0, 1.0, 4
    grad = torch.empty_like(v)
    torch.cuda.synchronize()
    loss, want = ctx.adjoint(st, v, [30.0], target, grad=grad)
    want = want.clone()
    with torch.cuda.stream(torch.cuda.Stream() if side_stream else torch.cuda.default_stream()):
        loss2, got = ctx.adjoint(st, late(torch, v), [30.0], late(torch, target), grad=grad)
    assert loss2 == loss and torch.equal(got, want)


def test_utr_images_and_volume(ctx, msk):
    """Also a volume that an earlier kernel is still writing."""
    torch = pytest.importorskip("torch")
    p = params(256, 64, 256)
    g = torch.Generator().manual_seed(2)
    im = (0.9 + 0.2 * torch.rand((12, 64, 256), generator=g)).cuda()
    ang = np.stack([np.zeros(12), np.linspace(0.0, 170.0, 12)], 1)
    run = lambda images, vol: ctx.utr_reconstruct(as_msk(msk, p), ang, np.full(12, 300.0), images, volume=vol)
    vol = torch.empty((256, 64, 256), device="cuda")
    torch.cuda.synchronize()
    want = run(im, vol).clone()
    torch.cuda.synchronize()
    got = run(late(torch, im), vol)
    # the sums of a voxel are added in any order
    assert float((got - want).norm() / want.norm()) < 1e-5
    torch.cuda.synchronize()
    torch.cuda._sleep(CYCLES)
    vol.zero_()
    got = run(im, vol)
    torch.cuda.synchronize()
    assert float((got - want).norm() / want.norm()) < 1e-5
