"""rode_sddmm's dense operands in every layout: what is row-major goes through as it is, other layouts are copied, the rest is refused."""
import pytest
import torch

from rode_b200.rode_sddmm import RoDeCSR, rode_sddmm, rode_sddmm_cuda

pytestmark = pytest.mark.gpu

LAYOUTS = {
    "row-major": lambda t: t,
    "column-major": lambda t: t.T.contiguous().T,
    "part of wider rows": lambda t: torch.cat([t, t], 1)[:, : t.shape[1]],
    "every second row": lambda t: torch.stack([t, -t], 1).reshape(-1, t.shape[1])[::2],
    "one row for all": lambda t: t[:1].expand(t.shape),
    "part of a buffer": lambda t: torch.cat([t[:2], t])[2:],
}


@pytest.mark.parametrize("layout", list(LAYOUTS))
def test_layouts(layout):
    S = RoDeCSR.from_random(200, 150, 9, torch.device("cuda"), k=32)
    lhs, rhs = torch.randn(200, 32, device="cuda"), torch.randn(150, 32, device="cuda")
    a, b = LAYOUTS[layout](lhs), LAYOUTS[layout](rhs)
    plain = [t.clone(memory_format=torch.contiguous_format) for t in (a, b)]
    fits = layout in ("row-major", "part of a buffer")
    assert rode_sddmm_cuda.sddmm_operands_fit(a, b, S.values, 200, 150, 32) is fits
    for x, y in ((a, b), (a, plain[1]), (plain[0], b)):
        assert torch.equal(rode_sddmm(S, x, y), rode_sddmm(S, *plain))


def test_what_is_refused():
    S = RoDeCSR.from_random(200, 150, 9, torch.device("cuda"), k=32)
    lhs, rhs = torch.randn(200, 32, device="cuda"), torch.randn(150, 32, device="cuda")
    for bad in (lhs[:199], lhs[:, :28], lhs[:, :, None], lhs.reshape(-1), torch.zeros(0, 32, device="cuda")):
        with pytest.raises(ValueError):
            rode_sddmm(S, bad, rhs)
    for bad in (rhs.half(), rhs.double(), rhs.int(), rhs.cpu()):
        with pytest.raises(AssertionError):
            rode_sddmm(S, lhs, bad)
