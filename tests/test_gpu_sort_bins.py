"""Track sort near its largest number of bins (GPU).

A sorted order's bins are one per action, two per material and one for idle slots; up to
384 fit the shared memory of the sort's blocks. Materials that no volume uses change no
track, so the transport must be that of the problem without them (energy depositions
are sums of FP64 atomics). More bins are refused with a message, before the first step;
orders that do not sort take any number of materials.
"""

import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MAX_BINS = 384


@pytest.fixture(scope="module")
def gb(built_lib):
    import celeritas_gb300 as gb

    gb.load_library(built_lib)
    return gb


def write_physics(gb, path, materials):
    """The calorimeter's physics with its first material (a vacuum) repeated."""
    with open(gb.physics_file("calo")) as f:
        lines = f.read().splitlines()
    num = int(next(ln for ln in lines if ln.startswith("materials ")).split()[2])
    first = [re.match(r"(material\.|(?:table|model|msc)\.(?:[^. ]+\.)+)0(\.[^ ]* .*)", ln)
             for ln in lines]
    out = ["materials 1 %d" % materials if ln.startswith("materials ") else ln for ln in lines]
    for i in range(num, materials):
        out += [m[1] + str(i) + m[2] for m in first if m]
    path.write_text("\n".join(out) + "\n")
    return str(path)


def stepper(gb, tmp_path, order, bins_over):
    """A stepper with the most materials that MAX_BINS + bins_over bins take."""
    probe = gb.Params(gb.physics_file("calo"), "calo", field_tesla=(0.0, 0.0, 1.0), msc=True,
                      track_order=order)
    materials = (MAX_BINS + bins_over - 1 - len(probe.action_labels())) // 2
    physics = write_physics(gb, tmp_path / "physics.txt", materials)
    params = gb.Params(physics, "calo", field_tesla=(0.0, 0.0, 1.0), msc=True,
                       track_order=order)
    return gb.Stepper(params, 8192, seed=2)


def transport(st, tuning={}):
    from celeritas_gb300.primaries import pencil_beam

    st.set_tuning(**tuning)
    res = [st.step(pencil_beam(4, energy=200.0))] + st.run(max_steps=5000)
    return [(r.generated, r.queued, r.active, r.alive) for r in res], st.energy_deposition()


@pytest.mark.parametrize("order, tuning", [
    ("reindex_both_action", {}),
    ("reindex_both_action", {"sort_material": 3}),
    ("reindex_step_limit_action", {}),
    ("reindex_particle_type", {}),
])
@pytest.mark.parametrize("bins_over", [0, -6, -12])
def test_many_bins(gb, tmp_path, order, tuning, bins_over):
    plain = gb.Stepper(gb.Params(gb.physics_file("calo"), "calo", field_tesla=(0.0, 0.0, 1.0),
                                 msc=True), 8192, seed=2)
    steps, edep = transport(plain)
    many_steps, many_edep = transport(stepper(gb, tmp_path, order, bins_over), tuning)
    assert many_steps == steps
    # Sums of at most ~10^5 FP64 terms in another order
    np.testing.assert_allclose(many_edep, edep, rtol=1e-10)


@pytest.mark.parametrize("graph_first", [False, True])
def test_too_many_bins(gb, tmp_path, graph_first):
    from celeritas_gb300.primaries import pencil_beam

    st = stepper(gb, tmp_path, "reindex_both_action", 2)
    if graph_first:
        with pytest.raises(gb.GbxError, match="at most 384"):
            st.step_kernels()
    with pytest.raises(gb.GbxError, match="at most 384"):
        st.step(pencil_beam(4, energy=200.0))
    with pytest.raises(gb.GbxError, match="at most 384"):
        st.step()
    # Without the sort the same stepper transports the primaries, still in wait
    st.set_tuning(sort=0)
    assert st.step().active == 4
    assert st.run(max_steps=5000)[-1].alive == 0
    unsorted_steps, _ = transport(stepper(gb, tmp_path, "none", 200))
    assert len(unsorted_steps) > 1
