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
