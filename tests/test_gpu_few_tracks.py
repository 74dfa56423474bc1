"""Charged along-step of few and many tracks in a field (GPU).

How the tracks are laid over the warps depends on how many there are: a warp (and
in the FP64 build the lanes of a warp) per track up to eight per SM, then up to 31
per warp, then consecutive tracks in consecutive lanes. With per-track random
streams a primary's steps do not depend on the others, so the first primaries of a
large batch end where they end on their own, bit for bit.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEPT = 24
STEPS = 4


@pytest.fixture(scope="module")
def gb(built_lib):
    import celeritas_gb300 as gb
    from celeritas_gb300.build import build

    gb.load_library(built_lib)
    gb.load_library(build(precision="mixed"), precision="mixed")
    return gb


@pytest.fixture(scope="module")
def sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


def kept_tracks(gb, params, prim, tuning):
    st = gb.Stepper(params, 2 * len(prim) + 100, seed=5)
    st.set_tuning(**tuning)
    st.step(prim)
    for _ in range(STEPS - 1):
        st.step()
    event, status = st.get_state("event_id", np.uint32), st.get_state("status", np.uint8)
    fields = [st.get_state("energy", params_real(st)), st.get_state("pos_x", np.float64),
              st.get_state("pos_z", np.float64), st.get_state("time", params_real(st, "time"))]
    slots = np.flatnonzero((status != 0) & (event < KEPT))
    rows = [(int(event[i]),) + tuple(float(f[i]) for f in fields) for i in slots]
    return sorted(rows)


def params_real(st, field="energy"):
    return np.float64 if st.state_info(field)[0] == 8 else np.float32


# Tracks per warp of 8 warps per SM: one, one and a bit, 31, 31 and a bit
@pytest.mark.parametrize("per_warp, more", [(1, 0), (1, 1), (31, 0), (31, 1)])
@pytest.mark.parametrize("precision, order, tuning", [
    ("double", "reindex_both_action", {}),
    ("double", "none", {}),
    ("double", "none", {"along_persistent": 1}),
    ("mixed", "reindex_both_action", {}),
    ("mixed", "reindex_particle_type", {"along_persistent": 0, "along_block_size": 128}),
])
def test_results_independent_of_track_count(gb, sms, precision, order, tuning, per_warp, more):
    from celeritas_gb300.workloads import eta_beam

    num = 8 * sms * per_warp + more
    params = gb.Params(gb.physics_file("cms"), "cms", field_tesla=(0.0, 0.0, 3.8), msc=True,
                       track_order=order, precision=precision, rng_per_track=True)
    prim = eta_beam(num, emin=0.5, emax=50.0, pdgs=(11, -11), eta_max=2.0, seed=9)
    # The kept primaries in events of their own, the others all in the next
    prim["event"] = np.minimum(np.arange(num), KEPT)
    few = kept_tracks(gb, params, prim[:KEPT], tuning)
    assert len(few) >= KEPT // 2
    assert kept_tracks(gb, params, prim, tuning) == few
