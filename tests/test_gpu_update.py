"""The cell update's variants and the grouped ghost pass at their edges.

* every rate regime of the cumulant update (omega_3 = omega_4 = 1 takes the
  variant without third-order moments) and the regularized-BGK update, in the
  one-CTA-per-block and the warp-specialised kernel, against the oracle: the
  single-step bar of test_gpu_stream_collide (2e-6 absolute, 1e-5 relative L2:
  a few rounding errors of the largest population);
* a density beyond the float range is stored as infinity, not as a large number;
* the ghost pass, paired and unpaired, on a refined region inside the domain and
  on domains whose edge cuts the blocks beyond that region, where a group of
  ring positions lies partly outside: bitwise the in-staging fill."""
import numpy as np
import pytest

from helpers import absent_neighbours, interior_refined_case, max_abs, rel_err, small_sphere_case

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from openludwig_b200 import _native as N  # noqa: E402
from openludwig_b200 import solver as S  # noqa: E402
from oracle import oracle as orc  # noqa: E402
from test_gpu_ws import _faults, _kernel, _one_step  # noqa: E402

DEV = torch.device("cuda:0")
AUTO, BLOCK, WS = 0, 1, 2

VARIANTS = [
    dict(name="omega3", op=0, limiter=1, omega_3=0.7),
    dict(name="omega4_fixed", op=0, limiter=1, adaptive_omega4=0, omega_4=1.2),
    dict(name="all_rates", op=0, limiter=2, omega_3=1.3, omega_4=0.8, omega_bulk=1.1, c_wale=0.5),
    dict(name="bgk", op=1),
    dict(name="bgk_wale_wall", op=1, c_wale=0.5, nu_sgs_bg=1e-4, wall_model=1),
    dict(name="bgk_o4_blend_turb", op=1, compressible=1, sponge_blend=1, inlet_turbulence=0.05),
]


@pytest.fixture(scope="module")
def sphere():
    return small_sphere_case(resolution=8)


@pytest.fixture(autouse=True)
def _policy():
    yield
    _kernel(AUTO)
    assert _faults() == 0


@pytest.mark.parametrize("choice,ctas", [(BLOCK, 0), (WS, 0), (WS, 7)],
                         ids=["block", "ws", "ws_7_ctas"])
@pytest.mark.parametrize("var", VARIANTS, ids=[v["name"] for v in VARIANTS])
def test_single_step_matches_oracle(sphere, var, choice, ctas):
    (f, r, v), inp = _one_step(sphere, var, choice, ctas)
    h = sphere[3][0]
    n = h.n_blocks
    o_f, o_rho = np.zeros(27 * 512 * n, np.float32), np.zeros(512 * n, np.float32)
    o_vel = np.zeros(3 * 512 * n, np.float32)
    orc.build()
    orc.stream_collide(dict(f_out=o_f, f_in=inp["f_in"], rho=o_rho, vel_out=o_vel,
                            vel_in=inp["vel_in"], obstacle=h.obstacle, sponge=h.sponge,
                            wall_dist=inp["wd"], neighbor_table=h.neighbor_table, map_x=h.map_x,
                            map_y=h.map_y, map_z=h.map_z, n_blocks=n), None,
                       {name: getattr(inp["sp"], name) for name, _ in N.STEP_FIELDS})
    assert max_abs(f, o_f) < 2e-6 and rel_err(f, o_f) < 1e-5
    assert max_abs(r, o_rho) < 2e-6 and max_abs(v, o_vel) < 2e-6


@pytest.mark.parametrize("choice", [BLOCK, WS], ids=["block", "ws"])
@pytest.mark.parametrize("value", [float("inf"), 3.2e38, float("-inf")])
@pytest.mark.parametrize("op", [0, 1], ids=["cumulant", "bgk"])
def test_density_out_of_range_is_stored(sphere, op, value, choice):
    c, mesh, p, hosts = sphere
    h = hosts[0]
    st = S.StepSettings(op=op, limiter=1, c_wale=0.5)
    cells = np.flatnonzero((np.asarray(h.obstacle).reshape(-1) == 0) &
                           (np.asarray(h.sponge).reshape(-1) == 0))[::97]
    _kernel(choice)
    lv = S.upload_level(h, DEV)
    src = lv.f_temp  # step 1 reads the second buffer
    src.view(27, -1)[13, torch.from_numpy(cells).to(DEV)] = value  # the rest population
    S.recursive_step([lv], st, 0, 1, None, 0.0, 0.05, (p.nx_coarse, p.ny_coarse, p.nz_coarse))
    got = lv.rho.cpu().numpy()[cells]
    # (the other 26 populations add 0.7, far below the last bit of 3.2e38)
    assert np.array_equal(got, np.full(len(cells), np.float32(max(value, 0.01))))


# Level-1 sizes: the refined region of the interior case ends at fine block
# (20, 18, 18), so fine blocks 21, 19 and 19 beyond it are cut by an edge at 2, 4
# and 6 of their 8 cells.
DOMAINS = {"edge": None, "inside": (0, 0, 0), "cut_x": (81, 0, 0), "cut_xyz": (81, 74, 75),
           "cut_yz": (0, 73, 73)}


@pytest.mark.parametrize("where", DOMAINS)
@pytest.mark.parametrize("ddf", [False, True], ids=["flow", "thermal"])
def test_ghost_pass_on_a_ragged_domain(ddf, where):
    kw = dict(compressibility_correction=True, ddf_enabled=True,
              u_target=np.float32(0.1)) if ddf else {}
    if where == "edge":  # the refined region reaches the domain's edge on all sides
        c, mesh, p, hosts = small_sphere_case(resolution=16, levels=2, c_wale=np.float32(0.5), **kw)
        dims = (p.nx_coarse - 1, p.ny_coarse - 2, p.nz_coarse - 5)
    else:
        c, mesh, p, hosts = interior_refined_case(**kw)
        dims = tuple(d or n for d, n in zip(DOMAINS[where],
                                            (p.nx_coarse, p.ny_coarse, p.nz_coarse)))
        inside, partly, outside = absent_neighbours(hosts[1], [2 * d for d in dims])
        assert inside > 5000 and (partly > 1000) == where.startswith("cut"), (inside, partly)
    st = S.StepSettings.from_config(c, False)
    runs = []
    for kind in ("paired", "unpaired", "none"):
        levels = [S.upload_level(h, DEV, ddf=ddf, ghost=kind != "none") for h in hosts]
        if kind == "unpaired":
            for lv in levels:
                lv.ghost2 = lv.ghost_g2 = None
        for t in range(1, 5):
            S.recursive_step(levels, st, 0, t, None, 0.0, 0.1 if ddf else 0.05, dims)
        torch.cuda.synchronize()
        runs.append(levels)
    assert runs[0][1].ghost2 is not None and runs[2][1].ghost is None
    for other in runs[:2]:
        for a, b in zip(other, runs[2]):
            assert torch.equal(a.f, b.f) and torch.equal(a.f_temp, b.f_temp)
            assert torch.equal(a.rho, b.rho) and torch.equal(a.vel, b.vel)
            if ddf:
                assert torch.equal(a.g, b.g) and torch.equal(a.g_temp, b.g_temp)
                assert torch.equal(a.temperature, b.temperature)
