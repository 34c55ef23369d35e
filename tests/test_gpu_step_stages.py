"""A step's graph runs chains of kernels beside one another and fuses routines;
stage replay runs every routine by itself, one after another. Every field of
the state is the same after both, bit for bit, so no chain misses what it
depends on and no fused routine computes something else. The optimized path's
Fourier fields between fused transforms are per-step scratch that
exogcm_step leaves unwritten in mode 1."""
import numpy as np
import pytest

from tests.helpers import oracle_field_list, pkg, planets

pytestmark = pytest.mark.gpu

STAGES = ("gridpointa", "spectrala", "physics_in", "fixer", "surface_flux", "radiation", "precipitation", "surface",
          "carbon", "storm", "physics_out", "spectrald", "pack")
SCRATCH = {1: {"fgt", "fgd", "fgz", "fgq", "fgp", "fgpj", "fdqt", "fzdekin"}}


def after_step_and_stages(mode, truncation, levels, slots, storm=False, change=None):
    """Fields that differ between a step and its stages."""
    whole, staged = (pkg.Engine(truncation, levels, slots, mode=mode) for _ in range(2))
    try:
        for e in (whole, staged):
            for s in range(slots):
                e.configure(s, planets.make_planet(91 + s % 2, truncation=truncation, levels=levels, stormclim=storm))
            e.step(3)
            e.step(4)
            if change:
                change(e)
        whole.step(1, publish_every=1)  # stage replay publishes
        for stage in STAGES:
            staged.run_stage(stage)
        names = [n for n in oracle_field_list() if n not in SCRATCH.get(mode, ())]
        return sorted({n for n in names for s in range(slots)
                       if not np.array_equal(whole.read(s, n), staged.read(s, n), equal_nan=True)})
    finally:
        whole.close()
        staged.close()


@pytest.mark.parametrize("mode,truncation,levels,slots,storm", [
    (0, 21, 5, 2, False), (0, 21, 10, 1, True), (1, 21, 5, 3, True), (1, 42, 10, 1, False),
    # more columns than the kernels with a thread per (column, level) take
    (1, 21, 10, 11, False), (1, 42, 5, 3, True),
    (2, 21, 10, 1, False), (2, 21, 5, 11, True), (2, 63, 5, 1, False)])
def test_step_equals_its_stages(mode, truncation, levels, slots, storm):
    assert after_step_and_stages(mode, truncation, levels, slots, storm) == []


@pytest.mark.parametrize("scale", [1e-34, 1e-36, 1e-38])
def test_step_equals_its_stages_at_tiny_humidity(scale):
    """Humidities around the smallest normal float, negative ones among them:
    the fixer flushes subnormals in a step as it does by itself."""

    def change(e):
        for name in ("sq", "sqm", "sqp"):
            e.write(0, name, (e.read(0, name).astype(np.float64) * scale).astype(np.float32))

    assert after_step_and_stages(1, 21, 10, 1, change=change) == []
