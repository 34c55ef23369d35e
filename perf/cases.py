"""The work this library is timed on: batches of model steps.

A case is one call as a program makes it on planets it has already admitted:
``Engine.step`` (or ``step_async``, or ``group_step`` over several engines) of
a few model steps. The range runs from one small planet stepped one step at a
time, as an interactive run does, to the ensembles whose throughput the
benchmark reports, over the three truncations, both level counts and the three
engine modes.

A pass advances the planets; its outputs are the state it leaves: the spectral
prognostic fields at both time levels and the temperatures and pressure of the
grid. Passes are one or a few steps long: a step costs the same in a batch of a
day's steps, and after a day two runs that round differently are two different
days' weather (a convective column more or less), while after a few steps they
are still the same.
"""
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("web-exoplasim_b200")
planets = importlib.import_module("web-exoplasim_b200.planets")

STEP_MINUTES = {21: 45.0, 42: 45.0, 63: 30.0}
LATITUDES = planets.LATITUDES

# Spectral prognostics at the new and the previous time level, then the
# temperatures of the air (with the surface's), the surface pressure, and the
# temperatures of the soil and the sea.
FIELDS = ("st", "sz", "sd", "sq", "sp", "stm", "szm", "sdm", "sqm", "spm", "dt", "dp", "dsoilt", "ysst")


def _case(name, truncation, levels, slots, mode, steps, call="step", publish=False, storm=False):
    return dict(name=name, truncation=truncation, levels=levels, slots=slots, mode=mode, steps=steps, call=call,
                publish=publish, storm=storm)


def listed():
    return [
        # The smallest call: one T21 L5 planet, a step at a time with its
        # snapshot published, as a page shows a run while it spins up.
        _case("one t21l5, plain, each step", 21, 5, 1, 0, 1, publish=True),
        # The single runs a page makes: the runner's engine (plain path, one slot).
        _case("one t42l10, plain", 42, 10, 1, 0, 2),
        # The same on the optimized path.
        _case("one t21l10", 21, 10, 1, 1, 4),
        _case("one t42l10", 42, 10, 1, 1, 2),
        # The single high-resolution run in split precision.
        _case("one t63l10, split", 63, 10, 1, 2, 2),
        # An odd handful of planets with the storm diagnostics on, publishing.
        _case("7 t42l5, storm", 42, 5, 7, 1, 1, publish=True, storm=True),
        # The blocks a server fills: T21 planets by the dozen, two batches in flight.
        _case("96 t21l5, async", 21, 5, 96, 1, 4, call="async"),
        _case("37 t21l10", 21, 10, 37, 1, 2),
        # Split precision on a batch.
        _case("48 t42l10, split", 42, 10, 48, 2, 1),
        # The high-resolution batch.
        _case("32 t63l10", 63, 10, 32, 1, 1),
        # The ensemble of the headline metric.
        _case("128 t42l10, async", 42, 10, 128, 1, 1, call="async"),
        # The mixed-resolution ensemble, one graph launch: T21 L5, T42 L10 and
        # T63 L10 planets in the proportion 4:3:1.
        _case("64+48+16 mixed", 0, 0, 16, 1, 1, call="group"),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    truncation = rng.choice((21, 21, 42, 42, 42, 63))
    levels = rng.choice((5, 10, 10))
    mode = rng.choice((0, 1, 1, 1, 1, 2))
    # at most the listed ensembles' cost; the plain path serves single runs and small batches
    most = {21: 192, 42: 96, 63: 32}[truncation] if mode else {21: 8, 42: 3, 63: 1}[truncation]
    slots = _log_int(rng, 1, most)
    steps = rng.choice((1, 1, 2))
    call = rng.choice(("step", "step", "async"))
    publish = rng.random() < 0.3
    storm = rng.random() < 0.1
    return dict(truncation=truncation, levels=levels, slots=slots, mode=mode, steps=steps, call=call, publish=publish,
                storm=storm)


def _planet(rng, truncation, levels, terrain, slot, storm):
    """A planet in a state a run passes through: a warm, half-saturated
    troposphere over a sea with a meridional gradient and ice at its cold end,
    from which winds, clouds, convection and rain set in within hours."""
    nlat = LATITUDES[truncation]
    nlon = 2 * nlat
    cfg = dict(terrain.config)
    cfg.update(fluxWm2=float(rng.uniform(0.97, 1.03) * 1367.0), co2Ppm=float(rng.uniform(250.0, 600.0)),
               obliquityDeg=float(rng.uniform(15.0, 30.0)), stormclim=storm)
    shift = int(rng.integers(nlon))

    def turned(field):
        return np.roll(np.asarray(field).reshape(nlat, nlon), shift, axis=1).reshape(-1)

    lat2 = np.repeat(planets.gaussian_sines(nlat) ** 2, nlon)
    sst = np.maximum(301.0 - 31.0 * lat2, 271.5)
    ice = (sst < 272.0).astype(np.float64)
    sigma = planets.sigma_levels(levels)
    t = (300.0 - 32.0 * lat2)[None, :] * sigma[:, None] ** 0.19
    t = np.maximum(t, 205.0) + 0.5 * rng.standard_normal((levels, nlat * nlon))
    p = sigma[:, None] * cfg["pressureBar"] * 1e5
    q = np.minimum(0.5 * planets.saturation(t, p, cfg["gasConstant"]), 0.015)
    q *= np.clip(sigma / 0.5, 0.02, 1.0)[:, None]  # drier aloft
    boundary = {172: turned(terrain.boundary[172]), 129: turned(terrain.boundary[129]), 169: sst, 210: ice}
    return planets.Planet(config=cfg, land_fraction=terrain.land_fraction, boundary=boundary, t_grid=t, q_grid=q,
                          seed=slot)


def _engine(case, truncation, levels, slots, seed):
    rng = np.random.default_rng([seed, truncation, levels, slots])
    terrains = [planets.make_planet(int(rng.integers(1 << 30)), truncation=truncation, levels=levels,
                                    timestepMinutes=STEP_MINUTES[truncation]) for _ in range(min(slots, 2))]
    e = pkg.Engine(truncation, levels, slots, mode=case["mode"])
    for s in range(slots):
        e.configure(s, _planet(rng, truncation, levels, terrains[s % len(terrains)], s, case["storm"]))
    e.step(3)  # the start-up steps
    return e


class _View:
    """A field of an engine, which stays alive as long as the tensor made from it."""

    def __init__(self, engine, field):
        self.engine = engine
        pointer, n = engine.device_field(field)
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (pointer, False), "version": 3,
                                         "strides": None}


def _state_of(e):
    """The engine's own buffers as tensors."""
    return {f: torch.as_tensor(_View(e, f), device="cuda") for f in FIELDS}


def prepare(case, seed):
    if case["call"] == "group":
        n = case["slots"]
        engines = [_engine(case, 21, 5, 4 * n, seed), _engine(case, 42, 10, 3 * n, seed),
                   _engine(case, 63, 10, n, seed)]
    else:
        engines = [_engine(case, case["truncation"], case["levels"], case["slots"], seed)]
    return dict(case=case, engines=engines, out=[_state_of(e) for e in engines])


def run(state):
    case, engines = state["case"], state["engines"]
    steps = case["steps"]
    if case["call"] == "group":
        pkg.group_step(engines, [steps] * len(engines))
    elif case["call"] == "async":
        engines[0].step_async(steps, publish_every=steps if case["publish"] else None)
    else:
        engines[0].step(steps, publish_every=steps if case["publish"] else None)
    return state["out"]


def _planet_step(truncation, levels):
    """Bytes and operations one planet's step cannot do without: the state
    read and written once (10 spectral prognostics and about 37 grid fields),
    the Legendre sums and FFTs of its transforms, and about 400 operations per
    grid point and level of column physics and grid-point dynamics."""
    nlat = LATITUDES[truncation]
    ntp1 = truncation + 1
    ncsp = ntp1 * (ntp1 + 1) // 2
    nhor = 2 * nlat * nlat
    nbytes = 4 * 2 * ((8 * levels + 2) * 2 * ncsp + (7 * levels + 36) * nhor)
    # a contraction: 2 (re, im) x NLAT / 2 x NCSP multiply-adds by latitude symmetry
    legendre = (48 * levels + 4) * 2 * 2 * (nlat // 2) * ncsp
    fft = (34 * levels + 5) * nlat * 2.5 * 2 * nlat * math.log2(2 * nlat)
    return nbytes, legendre + fft + 400.0 * levels * nhor


def work(case):
    if case["call"] == "group":
        n, k = case["slots"], case["steps"]
        parts = [(21, 5, 4 * n, k), (42, 10, 3 * n, k), (63, 10, n, k)]
    else:
        parts = [(case["truncation"], case["levels"], case["slots"], case["steps"])]
    nbytes = flops = 0.0
    for truncation, levels, slots, steps in parts:
        b, f = _planet_step(truncation, levels)
        nbytes += b * slots * steps
        flops += f * slots * steps
    return {"bytes": nbytes, "flops": flops}


def exact(case, seed):
    # The whole model has no short restatement in plain numpy.
    return None
