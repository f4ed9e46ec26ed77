"""Non-'over' composition modes (CUDA kernels behind compose_strokes) against the
float64 restatement of the reference's torch code (oracle.strokefield.compose_mode):
outputs within 1e-5, gradients of alphas, colours and density parameters within 1e-4
(helpers tolerances), both colour dimensions, batched leading shape."""
import pytest
import torch

from helpers import FWD_TOL, GRAD_TOL, rel
from neural3dstrokes_b200.strokes import compose_strokes
from oracle import strokefield as sf

pytestmark = pytest.mark.gpu

MODES = ["max", "max_density_weighted", "softmax", "softmax_density_weighted"]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("C,S", [(3, 37), (1, 5), (3, 300)])
def test_compose_mode_matches_reference_torch(cuda, mode, C, S):
    g = torch.Generator().manual_seed(S + C)
    a = torch.rand(6, 50, S, generator=g) ** 2
    c = torch.rand(6, 50, S, C, generator=g)
    d = torch.rand(S, generator=g) * 10
    gd = torch.randn(6, 50, generator=g)
    gc = torch.randn(6, 50, C, generator=g)
    ta, tc, td = (t.to(cuda).requires_grad_(True) for t in (a, c, d))
    dens, col = compose_strokes(ta, tc, td, mode)
    ((dens * gd.to(cuda)).sum() + (col * gc.to(cuda)).sum()).backward()
    ra, rc, rd = (t.double().requires_grad_(True) for t in (a, c, d))
    dens_r, col_r = sf.compose_mode(ra, rc, rd, mode)
    ((dens_r * gd.double()).sum() + (col_r * gc.double()).sum()).backward()
    assert rel(dens, dens_r) < FWD_TOL and rel(col, col_r) < FWD_TOL
    assert rel(ta.grad, ra.grad) < GRAD_TOL, rel(ta.grad, ra.grad)
    assert rel(tc.grad, rc.grad) < GRAD_TOL
    assert rel(td.grad, rd.grad) < GRAD_TOL, rel(td.grad, rd.grad)


def test_max_picks_first_of_ties(cuda):
    a = torch.tensor([[0.5, 0.9, 0.9, 0.1]], device=cuda)
    c = torch.arange(12, dtype=torch.float32, device=cuda).reshape(1, 4, 3)
    d = torch.ones(4, device=cuda)
    dens, col = compose_strokes(a, c, d, "max")
    assert float(dens[0]) == pytest.approx(0.9) and col[0].tolist() == [3.0, 4.0, 5.0]


def test_unknown_mode_raises(cuda):
    with pytest.raises(ValueError):
        compose_strokes(torch.rand(2, 3, device=cuda), torch.rand(2, 3, 3, device=cuda), torch.rand(3, device=cuda),
                        "median")


@pytest.mark.parametrize("S", [1, 31, 32, 33, 64, 65, 128, 129, 192, 193, 256, 257])
@pytest.mark.parametrize("mode", ["softmax", "softmax_density_weighted"])
def test_softmax_modes_at_register_edges(cuda, mode, S):
    """Forward and gradients against float64 at the stroke counts where the register
    kernels change (257: the general one). Tolerances: 1e-5 and 1e-4."""
    from neural3dstrokes_b200 import strokes as st_api
    g = torch.Generator().manual_seed(S)
    a, c, d = torch.rand(37, S, generator=g), torch.rand(37, S, 3, generator=g), torch.rand(S, generator=g) + 0.5
    gd, gc = torch.randn(37, generator=g), torch.randn(37, 3, generator=g)
    ours = [t.to(cuda).requires_grad_(True) for t in (a, c, d)]
    out = st_api.compose_strokes(*ours, mode)
    got = torch.autograd.grad(out, ours, (gd.to(cuda), gc.to(cuda)))
    ref = [t.double().requires_grad_(True) for t in (a, c, d)]
    key = ref[0] * ref[2] if mode == "softmax_density_weighted" else ref[0]
    w = torch.softmax(key / 0.05, -1)
    want = ((w * ref[0] * ref[2]).sum(-1), (w[..., None] * ref[1]).sum(-2))
    for x, y in zip(out, want):
        assert rel(x, y) < 1e-5
    for x, y in zip(got, torch.autograd.grad(want, ref, (gd.double(), gc.double()))):
        assert rel(x, y) < 1e-4


@pytest.mark.parametrize("S,C", [(1, 3), (33, 1), (128, 3), (256, 3), (260, 1), (1000, 3)])
@pytest.mark.parametrize("grad_mode", ["exact", "compat"])
def test_compose_backward_write_equals_accumulation(cuda, grad_mode, S, C):
    """The writing compose backward fills what the accumulating one adds to zeros, in the
    vector, row and compat kernels, whatever the buffers held."""
    from neural3dstrokes_b200 import strokelib as sl
    g = torch.Generator().manual_seed(S)
    a, c, d = (torch.rand(*s, generator=g).to(cuda) for s in ((53, S), (53, S, C), (S,)))
    gd, gc = torch.randn(53, generator=g).to(cuda), torch.randn(53, C, generator=g).to(cuda)
    before = sl.get_grad_mode()
    sl.set_grad_mode(grad_mode)
    try:
        want = [torch.zeros_like(t) for t in (a, c, d)]
        sl.compose_backward(*want, gd, gc, a, c, d)
        got = [torch.full_like(a, float("nan")), torch.full_like(c, float("nan")), torch.zeros_like(d)]
        sl._compose_backward("n3ds_compose_backward_write", *got, gd, gc, a, c, d)
    finally:
        sl.set_grad_mode(before)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert rel(got[2], want[2]) < 1e-6
