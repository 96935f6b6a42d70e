"""MLEM's voxel-driven update with detector columns interpolated in shared memory: each number
of slices per lane, one and two groups of rows more than the image holds, images shorter than
a chunk's rows, volumes that leave the image at its top, bottom and sides, off-centre
detectors, two chunks of slices, and values that are not finite; against FP64.  Positions of
up to 250 rows are good to about two units in the last place of FP32, 3e-5 rows, between taps
that differ by about their mean: 3e-5 relative L2.  (Voxels within 1e-3 pixels of the image's
edge in some view, which may fall to either side, are left out.)"""
import math

import pytest

from conftest import small_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from recon_b200 import BP_VOXEL, Options, Plan  # noqa: E402


def cfg(x, y, z, nv, nu, vox, pitch, **more):
    return small_cfg(Xdim=x, Ydim=y, Zdim=z, TAxPixels=nv, AxPixels=nu, XVoxSize=vox, YVoxSize=vox, ZVoxSize=vox,
                     TAxPixDim=pitch, AxPixDim=pitch, **{"NumProj": 35, "DeltaAng": 10.0, **more})


GEOMS = {f"slots{s}": cfg(9, 6, 32 * s - 5, 32 * s + 40, 40, 0.5, 1.0) for s in range(1, 9)}
GEOMS |= {f"group_more{s}": cfg(7, 10, 32 * s, 32 * s + 40, 40, 0.62, 1.0) for s in (2, 5, 8)}
GEOMS |= {
    "two_chunks": cfg(10, 9, 300, 250, 40, 0.4, 0.8),
    "short_image": cfg(12, 11, 160, 131, 50, 0.5, 1.0),       # as many groups as the image holds, the last in part
    "shorter_image": cfg(12, 11, 160, 100, 50, 0.5, 1.0),     # too short for the kernel
    "beyond_sides": cfg(60, 50, 60, 70, 40, 0.5, 1.0),
    "off_centre": cfg(20, 21, 64, 75, 60, 0.5, 1.0, Dx=3.3, Dz=-4.7),
    "dense_rows": cfg(20, 21, 64, 200, 60, 0.5, 0.45),        # the kernel for dense rows
}


def projected(P, c):
    """(u, v) of every voxel centre at every view in FP64, [view][z][y][x]."""
    axes = [(torch.arange(n, device="cuda", dtype=torch.float64) - (n - 1) / 2) * v
            for n, v in ((c["Zdim"], c["ZVoxSize"]), (c["Ydim"], c["YVoxSize"]), (c["Xdim"], c["XVoxSize"]))]
    z, y, x = torch.meshgrid(*axes, indexing="ij")
    for n in range(P.nproj):
        t = math.radians(P.angle(n))
        xa, ya = x * math.cos(t) - y * math.sin(t), x * math.sin(t) + y * math.cos(t)
        inv = c["Ry"] / (ya + c["Rf"])
        yield ((xa * inv - c["Dx"]) / (c["AxPixDim"] * c["M"]) + (P.nu - 1) / 2,
               (z * inv - c["Dz"]) / (c["TAxPixDim"] * c["M"]) + (P.nv - 1) / 2)


def update(P, c, f0, ratio):
    """f0 * Ht(ratio) / Ht(1) in FP64, and the voxels that lie clear of every image's edge."""
    ht, sens = torch.zeros_like(f0, dtype=torch.float64), torch.zeros_like(f0, dtype=torch.float64)
    clear = torch.ones_like(f0, dtype=torch.bool)
    for n, (u, v) in enumerate(projected(P, c)):
        inside = (u >= 0) & (u <= P.nu - 1) & (v >= 0) & (v <= P.nv - 1)
        for p, top in ((u, P.nu - 1), (v, P.nv - 1)):
            clear &= (p.abs() > 1e-3) & ((p - top).abs() > 1e-3)
        i, j = u.floor().clamp(0, P.nu - 2).long(), v.floor().clamp(0, P.nv - 2).long()
        a, b, img = u - i, v - j, ratio[n].double()
        val = (img[j, i] * (1 - a) + img[j, i + 1] * a) * (1 - b) + (img[j + 1, i] * (1 - a) + img[j + 1, i + 1] * a) * b
        ht += torch.where(inside, val, 0.0)
        sens += inside
    return torch.where(sens > 0, f0.double() * ht / sens.clamp(min=1), 0.0), clear


@pytest.mark.parametrize("name", list(GEOMS))
def test_staged_update(name):
    c = GEOMS[name]
    P = Plan(c, Options(bp=BP_VOXEL))
    gen = torch.Generator("cuda").manual_seed(611)
    f0 = torch.rand(P.shape_vol, device="cuda", generator=gen) + 0.5
    hf = P.fp_views(f0)
    g = torch.rand(hf.shape, device="cuda", generator=gen) * hf
    f = f0.clone()
    P.mlem_prepare()
    P.mlem_iteration(g, f)
    ratio = torch.where(hf != 0, g / hf, 0.0)
    want, clear = update(P, c, f0, ratio)
    assert clear.float().mean() > 0.9 and want[clear].abs().max() > 0
    assert ((f - want)[clear].norm() / want[clear].norm()).item() < 3e-5
    # an infinite ratio reaches the voxels that sample it, as an infinity or as a NaN
    at = (3, P.nv // 2, P.nu // 2)
    if hf[at] > 0:
        bad = g.clone()
        bad[at] = math.inf
        f = f0.clone()
        P.mlem_iteration(bad, f)
        u, v = list(projected(P, c))[at[0]]
        du, dv = (u - at[2]).abs(), (v - at[1]).abs()
        near, far = (du < 0.999) & (dv < 0.999), (du > 1.001) | (dv > 1.001)
        assert not torch.isfinite(f[near]).any()
        assert torch.isfinite(f[far]).all()
