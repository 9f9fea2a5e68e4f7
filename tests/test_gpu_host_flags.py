"""Rotation flags that travel as kernel arguments against flags on the device, and the one-launch column
weights against the elementwise form."""

import pytest
import torch

from helpers import activations, gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [16, 48, 512, 528, 4112])
@pytest.mark.parametrize("dtype", [torch.uint8, torch.bool])
def test_flags_from_the_host_and_from_the_device(k, dtype):
    from hi2_b200.format import fwht_groups
    from hi2_b200.hessian import transform_sigma

    flags = torch.randint(0, 2, (k // 16,), generator=gen(k)).to(dtype)
    if dtype == torch.uint8:
        flags = flags * 7  # anything that is not zero
    x = torch.randn(5, k, generator=gen(k + 1)).cuda()
    assert torch.equal(fwht_groups(x, flags), fwht_groups(x, flags.cuda()))
    sigma = (x.T @ x).contiguous()
    s16 = (0.5 + torch.rand(k, generator=gen(k + 2))).half().cuda()
    for a, b in zip(transform_sigma(sigma, s16, flags, 3.0, True), transform_sigma(sigma, s16, flags.cuda(), 3.0, True)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("k", [16, 240, 272, 4096, 4112])
@pytest.mark.parametrize("flagged", [None, "some"])
@pytest.mark.parametrize("scaled", [False, True])
def test_column_weights(k, flagged, scaled):
    from hi2_b200.stats import ColumnStats

    st = ColumnStats(k, "cuda")
    st.update(activations(200, k, k).cuda())
    flags = None if flagged is None else torch.randint(0, 2, (k // 16,), generator=gen(k)).to(torch.uint8)
    inv = (0.5 + torch.rand(k, generator=gen(k))).cuda() if scaled else None
    got = st.diag(flags, inv)
    m = (st.S / st.n).cpu()
    if scaled:
        v = inv.double().cpu().reshape(-1, 16)
        m = m * v[:, :, None] * v[:, None, :]
    h = torch.tensor([[(-1.0) ** bin(i & j).count("1") for j in range(16)] for i in range(16)], dtype=torch.float64) / 4
    plain, turned = m.diagonal(dim1=1, dim2=2), (h @ m @ h).diagonal(dim1=1, dim2=2)
    want = plain if flags is None else torch.where(flags[:, None] != 0, turned, plain)
    # 256 products in fp64 around the largest of them, then one rounding to fp32
    bound = 256 * 2.0**-53 * m.abs().amax((1, 2))[:, None] * 16 + 2.0**-24 * want.abs()
    assert bool(((got.cpu().double().reshape(-1, 16) - want).abs() <= bound).all())
