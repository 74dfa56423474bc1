"""Action sort over states of many sizes (GPU).

The sort's blocks take 1024 slots each, and the scan of a bin's block counts gives a
thread more than one of them beyond 1024 blocks. With per-track random streams the
transport is the same in any order of the slots, so each size must give the
unsorted state's steps and energy depositions (sums of FP64 atomics).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb(built_lib):
    import celeritas_gb300 as gb

    gb.load_library(built_lib)
    return gb


def transport(gb, order, slots):
    from celeritas_gb300.workloads import eta_beam

    params = gb.Params(gb.physics_file("cms"), "cms", field_tesla=(0.0, 0.0, 3.8), msc=True,
                       track_order=order, precision="double", rng_per_track=True)
    st = gb.Stepper(params, slots, seed=3)
    prim = eta_beam(6, emin=20.0, emax=100.0, pdgs=(11, 22), eta_max=1.5, seed=4)
    res = [st.step(prim)] + st.run(max_steps=5000)
    return [(r.generated, r.queued, r.active, r.alive) for r in res], st.energy_deposition()


@pytest.mark.parametrize("slots", [1023, 1024, 1025, 1 << 20, (1 << 20) + 1, (1 << 21) + 1025])
def test_sorted_transport_equals_unsorted(gb, slots):
    steps, edep = transport(gb, "none", slots)
    sorted_steps, sorted_edep = transport(gb, "reindex_both_action", slots)
    assert sorted_steps == steps
    # Sums of at most ~10^5 FP64 terms in another order
    np.testing.assert_allclose(sorted_edep, edep, rtol=1e-10)
