"""The launch shapes a step chooses by the size of the batch change no bit of
a planet's result: sizes on both sides of each line (columns per launch for
the kernels with a thread per (column, level) and for early launches, rows per
DFT chunk, runs per block of the dissipative heating's mean, tiles that end at
a field's last plane), in every mode, with empty slots between the planets."""
import numpy as np
import pytest

from tests.helpers import field_names, pkg, planets
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,truncation,levels,slots", [
    (1, 21, 10, 4), (1, 21, 10, 5), (1, 21, 10, 10), (1, 21, 10, 11), (1, 21, 5, 13), (1, 21, 10, 26), (1, 21, 10, 27),
    (1, 21, 10, 119), (1, 42, 10, 3), (1, 42, 5, 59), (1, 63, 5, 3),
    (0, 21, 5, 3), (0, 21, 10, 11), (0, 42, 10, 7),
    (2, 21, 5, 3), (2, 21, 10, 11), (2, 63, 10, 3)])
def test_planet_is_the_same_in_any_batch(mode, truncation, levels, slots):
    a = planets.make_planet(51, truncation=truncation, levels=levels)
    b = planets.make_planet(52, truncation=truncation, levels=levels, rotationPeriodDays=2.0, co2Ppm=3000.0)
    batch = pkg.Engine(truncation, levels, slots, mode=mode)
    alone = pkg.Engine(truncation, levels, 1, mode=mode)
    try:
        for s in range(0, slots, 2):
            batch.configure(s, b)
        batch.configure(slots - 1, a)
        alone.configure(0, a)
        for n in (1, 6):
            batch.step(n)
            alone.step(n)
        for name in field_names(oracle.Oracle(oracle.model_for(a))):
            x, y = batch.read(slots - 1, name), alone.read(0, name)
            assert np.array_equal(x, y, equal_nan=True), name
    finally:
        batch.close()
        alone.close()
