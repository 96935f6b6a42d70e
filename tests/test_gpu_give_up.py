"""A wait inside a kernel that runs out (a barrier that nothing completes, a limit of a few
milliseconds) reaches the caller as an error, once, and leaves the plan usable."""
import pytest

from conftest import small_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from recon_b200 import SIDDON_BP_GATHER, SIDDON_BP_RAY, Options, Plan, ReconError  # noqa: E402
from recon_b200._lib import check, lib  # noqa: E402

RECON_ERR_UNSUPPORTED, RECON_ERR_CUDA = 2, 3

CFG = small_cfg(Xdim=10, Ydim=10, Zdim=40, TAxPixels=66, NumProj=8, DeltaAng=45.0)


def _run_out(P):
    check(lib().recon_selftest_wait(P.handle, torch.cuda.current_stream().cuda_stream))


def test_reported_by_check_and_by_the_next_call():
    P = Plan(CFG, Options(siddon_bp=SIDDON_BP_GATHER))
    y = torch.rand((P.nproj, P.nv, P.nu), device="cuda", generator=torch.Generator("cuda").manual_seed(351))
    want = P.bp_views(y)
    P.check()
    _run_out(P)
    with pytest.raises(ReconError, match="ran out") as err:
        P.check()
    assert err.value.status == RECON_ERR_CUDA
    P.check()
    assert torch.equal(P.bp_views(y), want)
    _run_out(P)
    torch.cuda.synchronize()
    with pytest.raises(ReconError, match="ran out"):
        P.bp_views(y)
    assert torch.equal(P.bp_views(y), want)
    P.check()


def test_other_plans_have_no_waits():
    P = Plan(CFG, Options(siddon_bp=SIDDON_BP_RAY))
    with pytest.raises(ReconError) as err:
        _run_out(P)
    assert err.value.status == RECON_ERR_UNSUPPORTED
    P.check()


def test_each_plan_has_its_own_report():
    plans = [Plan(CFG, Options(siddon_bp=SIDDON_BP_GATHER)) for _ in range(3)]
    _run_out(plans[1])
    plans[0].check()
    plans[2].check()
    with pytest.raises(ReconError, match="ran out"):
        plans[1].check()
    _run_out(plans[1])
    plans[1].close()  # its word goes to the next plan, cleared
    again = Plan(CFG, Options(siddon_bp=SIDDON_BP_GATHER))
    for P in (plans[0], plans[2], again):
        P.check()
