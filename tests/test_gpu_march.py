"""A batch of coarse steps in one library call (ol_march) against the same
steps driven one level sub-step at a time (solver.recursive_step): the same
entry points with the same arguments, so every buffer is bitwise equal."""
import ctypes as C

import numpy as np
import pytest

from helpers import (absent_neighbours, interior_refined_case, interior_three_level_case,
                     small_sphere_case)

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from openludwig_b200 import _native as N  # noqa: E402
from openludwig_b200 import solver as S  # noqa: E402

DEV = torch.device("cuda:0")
DDF = dict(compressibility_correction=True, ddf_enabled=True, u_target=np.float32(0.1))
# "edge": the refined level fills the domain; "interior" (2 levels) and "three":
# refined levels inside it, whose values come from the parent's state
CASES = [
    dict(name="one_level", domain="one"),
    dict(name="refined", domain="edge", c_wale=np.float32(0.5), inlet_turbulence_intensity=0.02),
    dict(name="no_temporal", domain="edge", temporal_interpolation=False),
    dict(name="restriction", domain="edge", fine_to_coarse_restriction=True),
    dict(name="thermal", domain="edge", sponge_blend_distributions=True, **DDF),
    dict(name="interior", domain="interior"),
    dict(name="interior_no_temporal", domain="interior", temporal_interpolation=False),
    dict(name="interior_no_ghost", domain="interior", ghost=False),
    dict(name="interior_thermal", domain="interior", **DDF),
    dict(name="interior_thermal_restriction", domain="interior", fine_to_coarse_restriction=True,
         **DDF),
    dict(name="three", domain="three"),
    dict(name="three_no_temporal_restriction", domain="three", temporal_interpolation=False,
         fine_to_coarse_restriction=True),
    dict(name="three_thermal", domain="three", **DDF),
]


@pytest.fixture(scope="module")
def built():
    """A case's domain, built once for all its step counts."""
    made = {}

    def get(case):
        if case["name"] not in made:
            kw = {k: v for k, v in case.items() if k not in ("name", "domain", "ghost")}
            d = case["domain"]
            made.clear()  # (one case's domain at a time)
            made[case["name"]] = (interior_refined_case(**kw) if d == "interior" else
                                  interior_three_level_case(**kw) if d == "three" else
                                  small_sphere_case(resolution=8 if d == "one" else 16,
                                                    levels=1 if d == "one" else 2, **kw))
        return made[case["name"]]
    return get


@pytest.mark.parametrize("first,steps", [(1, 1), (1, 3), (4, 2), (-3, 4)])
@pytest.mark.parametrize("case", CASES, ids=[c["name"] for c in CASES])
def test_batch_equals_single_sub_steps(built, case, first, steps):
    c, mesh, p, hosts = built(case)
    st = S.StepSettings.from_config(c, False)
    dims, u = (p.nx_coarse, p.ny_coarse, p.nz_coarse), float(c.u_target)
    if case["domain"] in ("interior", "three"):
        assert len(hosts) == (3 if case["domain"] == "three" else 2)
        for i, h in enumerate(hosts[1:], 1):
            assert absent_neighbours(h, [d << i for d in dims])[0] > 5000
    runs = []
    for batch in (False, True):
        levels = [S.upload_level(h, DEV, ddf=c.ddf_enabled, ghost=case.get("ghost"))
                  for h in hosts]
        if batch:
            S.execute_timestep_batch(levels, st, first, steps, u, dims)
        else:
            for k in range(steps):
                S.recursive_step(levels, st, 0, first + k, None, 0.0, u, dims)
        torch.cuda.synchronize()
        runs.append(levels)
    names = ["f", "f_temp", "rho", "vel", "vel_temp"]
    names += ["g", "g_temp", "temperature"] if c.ddf_enabled else []
    old = ["f_old", "rho_old", "vel_old"] + (["g_old", "temperature_old"] if c.ddf_enabled else [])
    for i, (a, b) in enumerate(zip(*runs)):
        for n in names + (old if i + 1 < len(hosts) and st.use_temporal_interp else []):
            assert torch.equal(getattr(a, n), getattr(b, n)), (i, n)


def test_march_reports_bad_arguments():
    lv = (N.MarchLevel * 1)()
    with pytest.raises(N.OLError):
        N.call("ol_march", lv, 0, C.byref(N.StepParams()), None, 0, 8, 8, 8, 1, 1, None)
    with pytest.raises(N.OLError):  # thermal parameters without thermal buffers
        N.call("ol_march", lv, 1, C.byref(N.StepParams()), C.byref(N.ThermalParams()), 0, 8, 8, 8,
               1, 1, None)


@pytest.mark.parametrize("blocks", [1, 3, 97, 300])
def test_flow_statistics_of_any_block_count(blocks):
    g = torch.Generator(device=DEV).manual_seed(blocks)
    n = 512 * blocks
    rho = 1 + 0.1 * torch.randn(n, generator=g, device=DEV)
    vel = 0.1 * torch.randn(3 * n, generator=g, device=DEV)
    obs = (torch.rand(n, generator=g, device=DEV) < 0.3).to(torch.uint8)
    part = torch.empty(int(N.lib().ol_flow_stats_scratch_doubles(blocks)), dtype=torch.float64,
                       device=DEV)
    out = (C.c_double * 7)()
    N.call("ol_flow_stats", rho.data_ptr(), vel.data_ptr(), obs.data_ptr(), N.i32(blocks),
           part.data_ptr(), out, None)
    r, v2 = rho.double(), vel.double().reshape(3, n).square().sum(0)
    f = obs == 0
    want = [f.sum(), r[f].sum(), r[f].min(), r[f].max(), v2[f].max().sqrt(),
            (0.5 * r * v2)[f].sum(), r.sum()]
    # FP64 sums of up to 1.5e5 terms in another order: n * 2^-53 at most
    assert np.allclose(out[:], [float(w) for w in want], rtol=2e-11, atol=0)
