"""Force coefficients of the block pool, early in a run, against recorded ones.

While the start's pressure wave still runs, a body's drag swings through zero
and another rounding of one term of the cell update moves the coefficients by
1e-6 to 1e-2 of their vector.  The pool's cumulant update keeps one order and
rounding of its sums in every kernel form, so its coefficients repeat.  The
records (golden/pool_coefficients.json) are those of the update written with
the operators `/` and sqrtf and its sums in the order of the formulas; what is
left to differ is the order of the FP64 force sums, 1e-13 of their terms
(1e-10 where these cancel to a thousandth)."""
import dataclasses as dc
import json
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from openludwig_b200 import native, scaling, solver, workloads  # noqa: E402
from openludwig_b200.domain import setup_multilevel_domain  # noqa: E402

RECORDS = Path(__file__).parent / "golden" / "pool_coefficients.json"
STEPS = (120, 163)
# (body, finest cells, levels, Reynolds number, alpha, beta)
MIX = [("sphere", 16, 1, 3e4, 3.0, -2.0), ("cube", 24, 2, 1.5e5, 7.5, 1.0),
       ("sphere", 19, 3, 8e3, -1.0, 4.0)]
CASES = {
    "f32": dict(storage="f32"),
    "f16": dict(storage="f16"),
    "f32_rates": dict(storage="f32", omega_3=0.7, omega_4=1.1, omega_bulk=0.9, limiter=2),
    "f16_rates": dict(storage="f16", omega_3=1.2, adaptive_omega4=0, omega_4=0.9),
    "f32_thermal": dict(storage="f32", ddf=1, sponge_blend=1, compressible=1),
}


def pool_coefficients(storage, **settings):
    ddf = bool(settings.get("ddf"))
    ctx = native.Context(budget_bytes=1 << 30, storage=storage, ddf=ddf)
    ids = []
    for body, size, levels, re, alpha, beta in MIX:
        cfg, mesh = workloads.mix_case_config(workloads.MixCase(body, size, levels, re, alpha, beta))
        cfg = dc.replace(cfg, u_target=float(np.float32(0.05)), c_wale=0.5, ramp_steps=0)
        p = scaling.compute_domain_from_mesh(cfg, mesh.min_bounds, mesh.max_bounds)
        hosts = setup_multilevel_domain(cfg, mesh, p, device=0)
        if ddf:
            hosts = [dc.replace(h, tau_g=0.55) for h in hosts]
        st = dc.replace(solver.StepSettings.from_config(cfg, False), **settings)
        ids.append(ctx.add_case(native.PreparedCase(cfg, mesh, p, hosts, st)))
    out, done = [], 0
    for t in STEPS:
        ctx.step(t - done)
        done = t
        ctx.sync()
        out.append([list(ctx.coefficient_record(i).values()) for i in ids])
    ctx.close()
    return out


@pytest.mark.parametrize("name", CASES)
def test_pool_coefficients_repeat(name):
    got = np.array(pool_coefficients(**CASES[name]))
    want = np.array(json.loads(RECORDS.read_text())[name])
    assert got.shape == want.shape
    rel = np.linalg.norm(got - want, axis=2) / np.linalg.norm(want, axis=2)
    assert rel.max() < 1e-9, rel
