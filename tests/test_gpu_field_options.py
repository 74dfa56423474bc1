"""Field-driver options other than the default ones (GPU).

The FP64 build's transports equal the CPU restatement's step for step whatever the
options are: 'max_nsteps' from a chord search of one trial, whose last trial is
accepted or rejected by its error whatever its chord, to just below the 77 halvings
that the ~1e23 cm physics step of a near-vacuum takes, in a uniform field and in a
field map. In both builds a track's steps do not depend on how many others there are.
Depositions are sums of FP64 atomics in any order.
"""

import numpy as np
import pytest

from test_gpu_few_tracks import KEPT, kept_tracks

pytestmark = pytest.mark.gpu

TESLA = (0.0, 0.0, 3.8)


@pytest.fixture(scope="module")
def gb(built_lib):
    import celeritas_gb300 as gb
    from celeritas_gb300.build import build

    gb.load_library(built_lib)
    gb.load_library(build(precision="mixed"), precision="mixed")
    return gb


def source(gb, field):
    if field == "map":
        return {"rz_field": gb.field_map_file("cms")}
    return {"field_tesla": TESLA}


@pytest.mark.parametrize("field", ["uniform", "map"])
@pytest.mark.parametrize("max_nsteps", [1, 2, 3, 16, 75])
def test_transport_equals_restatement(gb, built_port, tmp_path, field, max_nsteps):
    import oracle
    from celeritas_gb300.primaries import write_primaries_text
    from celeritas_gb300.workloads import eta_beam

    slots, prim = 4096, eta_beam(6, emin=20.0, emax=500.0, pdgs=(11, 22), eta_max=1.5, seed=4)
    params = gb.Params(gb.physics_file("cms"), "cms", msc=True,
                       field_options={"max_nsteps": max_nsteps}, **source(gb, field))
    st = gb.Stepper(params, slots, seed=0)
    res = [st.step(prim)] + st.run(max_steps=20000)
    text = str(tmp_path / "primaries.txt")
    write_primaries_text(text, prim)
    extra = ["--msc", "--field-option", "max_nsteps", str(max_nsteps)]
    extra += (["--rz-field", gb.field_map_file("cms")] if field == "map"
              else ["--field"] + [repr(b) for b in TESLA])
    ref = oracle.run_port(gb.physics_file("cms"), text, slots, 0, geometry="cms", extra=extra)
    assert [(r.generated, r.queued, r.active, r.alive) for r in res] == ref["steps"]
    # At most ~10^5 deposits a volume, each sum's rounding 2^-53 of the total
    np.testing.assert_allclose(st.energy_deposition().sum(), sum(ref["edep"].values()),
                               rtol=1e-11)


# Tracks per warp of 8 warps per SM: one, one and a bit, 31 and a bit
@pytest.mark.parametrize("per_warp, more", [(1, 0), (1, 1), (31, 1)])
@pytest.mark.parametrize("precision, tuning, field, options", [
    ("double", {}, "uniform", {"max_nsteps": 1}),
    ("double", {}, "uniform", {"max_nsteps": 5, "delta_chord": 0.001}),
    ("double", {}, "map", {"max_nsteps": 16, "epsilon_rel_max": 1e-5}),
    ("double", {"along_block_size": 512}, "map", {}),
    ("mixed", {}, "map", {"max_nsteps": 3}),
])
def test_results_independent_of_track_count(gb, precision, tuning, field, options, per_warp,
                                            more):
    import torch
    from celeritas_gb300.workloads import eta_beam

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    num = 8 * sms * per_warp + more
    params = gb.Params(gb.physics_file("cms"), "cms", msc=True, precision=precision,
                       rng_per_track=True, field_options=options, **source(gb, field))
    prim = eta_beam(num, emin=0.5, emax=50.0, pdgs=(11, -11), eta_max=2.0, seed=9)
    # The kept primaries in events of their own, the others all in the next
    prim["event"] = np.minimum(np.arange(num), KEPT)
    few = kept_tracks(gb, params, prim[:KEPT], tuning)
    assert len(few) >= KEPT // 2
    assert kept_tracks(gb, params, prim, tuning) == few
