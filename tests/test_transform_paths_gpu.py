"""Forms of the flow's passes that a plan chooses by size, batch or alignment: they agree with the
forms that the oracle tests cover."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    assert torch.cuda.is_available()
    return torch


def _state(torch, p, seed, nbox=None):
    """A smooth random cube spectrum, the same for every precision."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = ((nbox,) if nbox else ()) + (3, p.Mx, p.My, p.Mzp)
    uk = torch.view_as_complex(torch.randn(shape + (2,), dtype=torch.float64, device="cuda", generator=g))
    k = torch.cat([torch.arange(p.kc + 1), torch.arange(-p.kc, 0)]).double().cuda()
    kz = torch.arange(p.Mzp).double().cuda()
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz ** 2
    uk = uk * torch.where(k2 <= p.kc * p.kc + p.kc, p.N ** 3 / (1.0 + k2), 0.0)
    return uk.to(p.cdtype)


# FP32 tolerance of one RHS evaluation (tests/test_dns_gpu.py)
TOL = 2e-5


@pytest.mark.parametrize("N", [64, 128, 256])
def test_state_off_the_16_byte_grid(torch, N):
    """A contiguous state that starts 8 bytes past a 16-byte boundary takes one column per thread and
    no row prefetch; the same RHS to FP32 rounding, and nothing past the end is read or written."""
    from lucky_droplets_b200.spectral import Plan
    p = Plan(N, "f32")
    uk = _state(torch, p, N)
    ref = p.velocity_rhs(uk, 0.01, 1.0, (1, 2))
    off = torch.zeros(uk.numel() + 1, dtype=uk.dtype, device="cuda")[1:].view(uk.shape)
    out = torch.zeros(uk.numel() + 1, dtype=uk.dtype, device="cuda")[1:].view(uk.shape)
    off.copy_(uk)
    assert off.data_ptr() % 16 == 8 and out.data_ptr() % 16 == 8
    got = p.velocity_rhs(off, 0.01, 1.0, (1, 2), ku=out)
    assert float(torch.linalg.norm(got - ref) / torch.linalg.norm(ref)) < TOL
    assert torch.equal(off, uk)


@pytest.mark.parametrize("N,nbox", [(64, 3), (64, 8), (32, 5), (16, 2)])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_boxes_of_a_batch_equal_boxes_alone(torch, N, nbox, prec):
    """The plane pass of few planes and of many (three blocks per SM from 444 planes of FP32 64)."""
    from lucky_droplets_b200.spectral import Plan
    many, one = Plan(N, prec, nbox=nbox), Plan(N, prec)
    uk = _state(torch, one, N + nbox, nbox)
    ku = torch.zeros_like(uk)
    many.velocity_rhs(uk, 0.01, 1.0, (1, 2), ku=ku)
    for b in range(nbox):
        assert torch.equal(ku[b], one.velocity_rhs(uk[b].contiguous(), 0.01, 1.0, (1, 2)))


@pytest.mark.parametrize("N", [384, 512])
def test_large_grids_fp32_against_fp64(torch, N):
    """Two columns per thread with three radix stages (512), the longest 12 R2 R3 rows (384)."""
    from lucky_droplets_b200.spectral import Plan
    p32 = Plan(N, "f32")
    uk = _state(torch, p32, N)
    got = p32.velocity_rhs(uk, 0.01, 1.0, (1, 2))
    p64 = Plan(N, "f64")
    ref = p64.velocity_rhs(uk.to(torch.complex128), 0.01, 1.0, (1, 2))
    assert float(torch.linalg.norm(got - ref) / torch.linalg.norm(ref)) < TOL
    assert np.isfinite(float(got.abs().max()))


@pytest.mark.parametrize("tuning", [None, [0, 0]])
def test_y_passes_of_more_planes_than_a_grid_dimension(torch, tuning):
    """683 boxes of 96^3 are 65,568 outer indices of the y passes, more than a second grid dimension
    takes: the same values as a box alone, whose y passes are one-shot tiles."""
    from lucky_droplets_b200.spectral import Plan
    torch.cuda.empty_cache()
    N, nbox = 96, 683
    many, one = Plan(N, "f64", nbox=nbox), Plan(N, "f64")
    if tuning:
        many.set_tuning(tuning)
    uk = torch.zeros((nbox, 3, one.Mx, one.My, one.Mzp), dtype=one.cdtype, device="cuda")
    for b in (0, nbox - 1):
        uk[b] = _state(torch, one, b)
    ku = torch.zeros_like(uk)
    many.velocity_rhs(uk, 0.01, 1.0, (1, 2), ku=ku)
    for b in (0, nbox - 1):
        assert torch.equal(ku[b], one.velocity_rhs(uk[b].contiguous(), 0.01, 1.0, (1, 2)))
    assert not torch.view_as_real(ku[1:-1]).any()


@pytest.mark.parametrize("N,prec,nbox", [(64, "f32", 1), (96, "f32", 1), (16, "f64", 4096)])
def test_autotune_where_the_plane_pass_runs(torch, N, prec, nbox):
    """Grids whose right-hand side takes the plane pass have no y pass to time."""
    from lucky_droplets_b200.spectral import Plan
    p = Plan(N, prec, nbox=nbox)
    assert p.autotune() == {"ms": {"inverse_y": [-1.0] * 4, "forward_y": [-1.0] * 4}, "choice": [0, 0]}


@pytest.mark.parametrize("N,prec", [(96, "f64"), (128, "f32"), (128, "f64"), (192, "f64"), (360, "f32")])
def test_y_pass_variants_give_identical_rhs(torch, N, prec):
    from lucky_droplets_b200.spectral import Plan
    p = Plan(N, prec)
    uk = _state(torch, p, N)
    ref = p.velocity_rhs(uk, 0.01, 1.0, (1, 2)).clone()
    for choice in ([0, 0], [1, 1], [3, 3]):
        p.set_tuning(choice)
        assert torch.equal(p.velocity_rhs(uk, 0.01, 1.0, (1, 2)), ref)


class _Guarded:
    """A tensor `off` bytes past a 16-byte boundary between two stretches of NaN."""

    def __init__(self, torch, shape, dtype, off):
        n, item = int(np.prod(shape)), torch.empty(0, dtype=dtype).element_size()
        self.torch, self.lo = torch, 64 + off // item
        self.hi = self.lo + n
        self.all = torch.full((self.hi + 64,), complex("nan+nanj"), dtype=dtype, device="cuda")
        self.t = self.all[self.lo:self.hi].view(shape)
        assert self.t.data_ptr() % 16 == off

    def intact(self):
        ends = self.torch.cat([self.all[:self.lo], self.all[self.hi:]])
        return bool(self.torch.isnan(self.torch.view_as_real(ends)).all())


@pytest.mark.parametrize("off", [(8, 8, 8), (0, 0, 8), (8, 0, 0), (0, 8, 0)])
@pytest.mark.parametrize("N", [64, 128, 256])
def test_stages_off_the_16_byte_grid_stay_inside(torch, N, off):
    """RK2 and RK4 stages and the right-hand side with the state, the stage state or the accumulator 8
    bytes past a 16-byte boundary: the values of aligned buffers to FP32 rounding, and nothing outside
    the buffers is written, or read and used."""
    import ctypes
    from lucky_droplets_b200 import _lib
    from lucky_droplets_b200._lib import check, ptr, stream_ptr
    from lucky_droplets_b200.spectral import Plan, flow_params
    p = Plan(N, "f32")
    uk = _state(torch, p, N)
    prm = ctypes.byref(flow_params(1e-3, 0.01, 1.0, (1, 2)))

    def stages(offs, call, count):
        bufs = [_Guarded(torch, uk.shape, uk.dtype, o) for o in offs]
        bufs[0].t.copy_(uk)
        for b in bufs[1:]:
            b.t.zero_()
        for s in range(1, count + 1):
            check(call(p.handle, s, *[ptr(b.t) for b in bufs], None, prm, stream_ptr(None)))
        assert all(b.intact() for b in bufs)
        return [b.t for b in bufs]

    L = _lib.lib()
    for call, count in ((L.ld_rk2if_stage, 2), (L.ld_rk4_stage, 4)):
        for got, ref in zip(stages(off, call, count), stages((0, 0, 0), call, count)):
            assert float(torch.linalg.norm(got - ref) / torch.linalg.norm(ref)) < TOL
    y, ku = (_Guarded(torch, uk.shape, uk.dtype, o) for o in off[:2])
    y.t.copy_(uk)
    p.velocity_rhs(y.t, 0.01, 1.0, (1, 2), ku=ku.t)
    ref = p.velocity_rhs(uk, 0.01, 1.0, (1, 2))
    assert y.intact() and ku.intact() and torch.equal(y.t, uk)
    assert float(torch.linalg.norm(ku.t - ref) / torch.linalg.norm(ref)) < TOL


# relative errors of FP32 against FP64 with rows of 8 x 8 x 2 and 8 x 8 x 4, which 16 x 8 and 16 x 16 replaced
@pytest.mark.parametrize("N,rhs,fft", [(128, 2.81e-7, 1.64e-7), (256, 3.40e-7, 1.82e-7)])
def test_rows_of_radix_16_are_no_less_accurate(torch, N, rhs, fft):
    from lucky_droplets_b200.spectral import Plan
    p, q = Plan(N, "f32"), Plan(N, "f64")

    def err(a, b):
        return float(torch.linalg.norm(a - b) / torch.linalg.norm(b))

    uk = _state(torch, p, N)
    assert err(p.velocity_rhs(uk, 0.01, 1.0, (1, 2)), q.velocity_rhs(uk.to(q.cdtype), 0.01, 1.0, (1, 2))) < rhs
    u = torch.randn((1, N, N, N), device="cuda", generator=torch.Generator(device="cuda").manual_seed(N))
    f = q.rfft_mpi(u.double())
    assert err(p.rfft_mpi(u), f) < fft
    f = f.to(p.cdtype)
    assert err(p.irfft_mpi(f), q.irfft_mpi(f.to(q.cdtype))) < fft
