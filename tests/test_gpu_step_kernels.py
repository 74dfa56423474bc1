"""Kernel launches of a graph-replayed step (GPU)."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb(built_lib):
    import celeritas_gb300 as gb
    from celeritas_gb300.build import build

    gb.load_library(built_lib)
    gb.load_library(build(precision="mixed"), precision="mixed")
    return gb


def test_counting_leaves_pending_primaries(gb):
    """Primaries in wait when the launches are counted enter the next step only."""
    from celeritas_gb300.primaries import pencil_beam

    params = gb.Params(gb.physics_file("calo"), "calo")

    def transport(count):
        st = gb.Stepper(params, 4096, seed=1)
        st.insert_primaries(pencil_beam(2, energy=100.0))
        if count:
            assert st.step_kernels() > 0
        res = [st.step()] + st.run(max_steps=2000)
        return [(r.generated, r.queued, r.active, r.alive) for r in res]

    steps = transport(False)
    assert steps[0][0] == 2 and steps[-1][3] == 0
    assert transport(True) == steps


# More than without a field: the FP64 build's kernel for few tracks, the list of the
# charged tracks where none is sorted, and the clearing of what the list and the
# persistent kernel count with
@pytest.mark.parametrize("precision, order, persistent, more", [
    ("double", "reindex_both_action", 0, 1),
    ("double", "reindex_both_action", 1, 1),
    ("double", "none", 0, 3),
    ("mixed", "reindex_both_action", 0, 0),
    ("mixed", "reindex_both_action", 1, 1),
    ("mixed", "none", 0, 2),
    ("mixed", "reindex_particle_type", 1, 2),
])
def test_launches_for_a_field(gb, precision, order, persistent, more):
    def kernels(field):
        params = gb.Params(gb.physics_file("calo"), "calo", field_tesla=(0.0, 0.0, field),
                           msc=True, track_order=order, precision=precision)
        st = gb.Stepper(params, 4096, seed=1)
        st.set_tuning(along_persistent=persistent)
        return st.step_kernels()

    assert kernels(1.0) - kernels(0.0) == more
