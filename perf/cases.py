"""The calls whose speed counts: what a user of this framework has it compute.

Each case is one pass through the public engines (``opengate_gb300.engine``) as a
simulation script drives them: reset, run, fetch the images.  The sizes span the
configurations of ``bench.py`` and of the tests, from the 64^3 water cube with a
few thousand primaries to the 256 x 256 x 160 CT with 1e8, and odd grids between.

A case is made from its dict and a seed.  The seed picks the histories (the
Philox key), the anatomy (the phantom rolled along z and mirrored) and, for the
network cases, the rows and the weights.  The phantom on which that is done and
the physics tables do not depend on the seed and are kept per size.
"""

import copy
import functools
import math

import numpy as np
import torch

from opengate_gb300 import _capi as C
from opengate_gb300 import materials as M
from opengate_gb300 import spect as S
from opengate_gb300 import tables as T
from opengate_gb300 import workloads as W
from opengate_gb300.engine import ArfNetwork, BatchEngine, DoseEngine, SpectEngine
from opengate_gb300.scene import Scene, SourceSpec

TC99M_WINDOWS = ((0.126, 0.154), (0.108, 0.126))
LU177_WINDOWS = ((0.1872, 0.2288), (0.166, 0.187), (0.1017, 0.1243))
HOUSING = "nm670"
WORLD = 1500.0
N_HEADS = 2
HID, OUT_PAD = 128, 16  # the ARF network: 3 -> 128 -> 128 -> 128 -> windows + 1 (16 padded)
N_PARAMS = HID * 3 + HID + 2 * (HID * HID + HID) + OUT_PAD * HID + OUT_PAD
THETA_MAX, E_RANGE, ROULETTE = 85.0, (0.1017, 0.21), 40.0  # the network's training domain


def listed():
    """The cases that are timed, by use: what each one stands for is said beside it."""
    return [
        # A first look at a small phantom, as scripts and the tests do: a pencil beam on the 64^3 water
        # cube, so few primaries that latency and launches decide; images fetched.
        dict(name="dose_preview", kind="dose", phantom="water", nx=64, ny=64, nz=64, spacing=2.0, energy=1.0,
             primaries=20_000, precision=32, grid=0, tle=0),
        # The headline: the CT phantom at full resolution, field source with a 60-bin spectrum to 6 MeV, edep
        # and edep^2 with 1e8 primaries; the largest ordinary dose run.
        dict(name="dose_ct", kind="dose", phantom="ct", nx=256, ny=256, nz=160, spacing=1.2, energy=6.0,
             primaries=100_000_000, precision=32, grid=0, tle=0),
        # A planning dose: an odd CT grid and a DoseActor with a coarser grid of its own (edep, dose and
        # their squares), partly outside the image.
        dict(name="dose_ct_grid", kind="dose", phantom="ct", nx=181, ny=143, nz=97, spacing=1.9, energy=6.0,
             primaries=5_000_000, precision=32, grid=3, tle=0),
        # The same path in FP64 arithmetic, the option a user takes to check a result.
        dict(name="dose_fp64", kind="dose", phantom="ct", nx=128, ny=128, nz=80, spacing=2.4, energy=6.0,
             primaries=1_000_000, precision=64, grid=0, tle=0),
        # TLEDoseActor: every crossed voxel scored, the variance-reduced dose of low-energy beams.
        dict(name="dose_tle", kind="dose", phantom="water", nx=64, ny=64, nz=64, spacing=2.0, energy=1.0,
             primaries=3_000_000, precision=32, grid=0, tle=1),
        # Many uneven simulations in one set of launches (slab phantoms of 32 to 128 voxels a side, 50 keV to
        # 2 MeV), replayed as a CUDA graph; all images fetched.
        dict(name="dose_batched", kind="batched", sims=24, primaries_lo=1e5, primaries_hi=1e7),
        # Tc-99m acquisition with a LEHR collimator, two heads, 60 positions, every photon tracked through
        # phantom, collimator and crystal; projections fetched.
        dict(name="spect_tc99m", kind="spect", recipe="plain", nuclide="tc99m", nx=256, ny=256, nz=160, spacing=1.2,
             runs=60, pixels=128, primaries=30_000_000),
        # The same acquisition by the free-flight recipe: forced-direction primaries plus scatter splitting
        # with 50 / 10 copies; weighted projections and their squares fetched.
        dict(name="spect_freeflight", kind="spect", recipe="ff", nuclide="tc99m", nx=128, ny=128, nz=80, spacing=2.4,
             runs=60, pixels=128, primaries=10_000_000),
        # Lu-177 with ARF detectors, 120 positions, three windows: the same recipe with 10 / 2 copies and the
        # network in the place of the heads.
        dict(name="spect_arf", kind="spect", recipe="arf", nuclide="lu177", nx=128, ny=128, nz=80, spacing=2.4,
             runs=120, pixels=128, primaries=50_000_000),
        # Training rows of the ARF network: photons tracked through the MELP head, all rows kept (the actor's
        # default, no Russian roulette) and fetched.
        dict(name="arf_dataset", kind="arf_dataset", collimator="melp", samples=1_000_000),
        # Training the network on given rows (forward and backward, Adam): the weights come back.
        dict(name="arf_train", kind="arf_train", rows=262_144, batch=8192, epochs=2),
        # Inference on host rows: probabilities of an odd number of photons.
        dict(name="arf_predict", kind="arf_predict", rows=1_000_003),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(("water", "ct", "grid", "fp64", "tle", "batched", "plain", "ff", "arf", "arf_dataset",
                       "arf_train", "arf_predict"))
    if kind in ("water", "tle"):
        n = int(_log(rng, 31, 129))
        return dict(kind="dose", phantom="water", nx=n, ny=n, nz=n, spacing=round(rng.uniform(1.0, 3.0), 2),
                    energy=round(_log(rng, 0.06, 6.0 if kind == "water" else 1.5), 3),
                    primaries=int(_log(rng, 5e3, 2e7 if kind == "water" else 4e6)), precision=32, grid=0,
                    tle=int(kind == "tle"))
    if kind in ("ct", "grid", "fp64"):
        top = {"ct": 6e7, "grid": 2e7, "fp64": 2e6}[kind]
        return dict(kind="dose", phantom="ct", nx=int(_log(rng, 64, 256)), ny=int(_log(rng, 64, 256)),
                    nz=int(_log(rng, 40, 160)), spacing=round(rng.uniform(1.2, 4.0), 2),
                    energy=round(_log(rng, 0.4, 6.0), 2), primaries=int(_log(rng, 1e4, top)),
                    precision=64 if kind == "fp64" else 32, grid=rng.randint(2, 5) if kind == "grid" else 0, tle=0)
    if kind == "batched":
        return dict(kind="batched", sims=rng.randint(2, 28), primaries_lo=1e4, primaries_hi=round(_log(rng, 1e5, 6e6)))
    if kind in ("plain", "ff", "arf"):
        top = {"plain": 4e7, "ff": 1.5e7, "arf": 8e7}[kind]
        return dict(kind="spect", recipe=kind, nuclide=rng.choice(("tc99m", "lu177")), nx=rng.randint(64, 160),
                    ny=rng.randint(64, 160), nz=rng.randint(40, 100), spacing=round(rng.uniform(2.2, 4.0), 2),
                    runs=rng.randint(4, 120), pixels=rng.randint(64, 128), primaries=int(_log(rng, 2e5, top)))
    if kind == "arf_dataset":
        return dict(kind="arf_dataset", collimator=rng.choice(("lehr", "melp")), samples=int(_log(rng, 2e4, 4e6)))
    if kind == "arf_train":
        return dict(kind="arf_train", rows=int(_log(rng, 3e4, 6e5)), batch=128 * rng.randint(8, 80),
                    epochs=rng.randint(1, 4))
    return dict(kind="arf_predict", rows=int(_log(rng, 500, 4e6)))


# ---- phantoms, tables and sources -------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _ct_materials(spect):
    """(HU intervals, label table, physics tables, number of CT materials); with the heads' materials for SPECT."""
    vm, lut, mats = W.ct_materials()
    extra = ["G4_Pb", "G4_SODIUM_IODIDE", *S.HOUSING_MATERIALS[HOUSING]] if spect else []
    db = M.MaterialDatabase()
    return vm, lut, T.PhysicsTables(mats + [db.get(m) for m in extra]), len(mats)


@functools.lru_cache(maxsize=8)
def _ct_image(nx, ny, nz, spacing, spect):
    """(labels, activity) of the CT phantom before the seed's mirror and roll."""
    vm, lut, _, _ = _ct_materials(spect)
    hu = W.ct_hu_image(shape=(nz, ny, nx), spacing=spacing)
    act = W.activity_phantom(hu, spacing) if spect and min(nx, ny) * spacing >= 250 and nz * spacing >= 90 else None
    if spect and act is None:
        act = (hu > -500).astype(np.float64)
    return M.create_label_image(hu, "G4_AIR", vm, lut), act


def _anatomy(image, seed):
    image = np.roll(image, int(seed) * 7 % image.shape[0], axis=0)
    return np.ascontiguousarray(image[:, :, ::-1] if seed & 1 else image)


def _corner(case):
    return [-case[k] * case["spacing"] / 2 for k in ("nx", "ny", "nz")]


def _field_source(case):
    """Point source at 1 m from the patient, a 10 x 10 cm field at the isocentre, E exp(-E / 1.5 MeV) spectrum."""
    src = SourceSpec()
    src.pos_type = C.GG_POS_POINT
    sad, field = 1110.0, 100.0
    src.translation = [0.0, -sad, 0.0]
    src.dir_type = C.GG_DIR_ISO
    half = math.atan(math.hypot(field / 2, field / 2) / sad)
    src.theta = [math.pi / 2 - half, math.pi / 2 + half]
    src.phi = [1.5 * math.pi - half, 1.5 * math.pi + half]
    y = _corner(case)[1] - 1.0
    hf = field / 2 * (y + sad) / sad
    src.accept_boxes = [((-hf, y - 0.5, -hf), (hf, y + 0.5, hf))]
    src.ene_type = C.GG_ENE_HISTOGRAM
    src.spec_e, src.spec_cdf = W.spectrum_e_exp(e_hi=case["energy"])
    return src


def _dose_scene(case, seed):
    if case["phantom"] == "water":
        scene = W.water_pencil(case["nx"], case["spacing"], case["energy"])
        src = copy.copy(scene.source)
        jitter = np.random.default_rng(seed).uniform(-0.4, 0.4, 2) * case["spacing"]
        src.translation = [float(jitter[0]), float(jitter[1]), src.translation[2]]
        scene.set_source(src)
        return scene
    labels = _anatomy(_ct_image(case["nx"], case["ny"], case["nz"], case["spacing"], False)[0], seed)
    return Scene(_ct_materials(False)[2], labels, [case["spacing"]] * 3, _corner(case), [WORLD] * 3, 0,
                 _field_source(case))


def _spect_scene(case, seed):
    """(scene, head and gantry specification) of a SPECT case."""
    labels, act = _ct_image(case["nx"], case["ny"], case["nz"], case["spacing"], True)
    _, _, pt, n_ct = _ct_materials(True)
    lines, yields = W.TC99M if case["nuclide"] == "tc99m" else W.LU177
    src = SourceSpec()
    src.set_activity_image(_anatomy(act, seed), [case["spacing"]] * 3, _corner(case))
    src.dir_type = C.GG_DIR_ISO
    src.ene_type = C.GG_ENE_LINES
    src.spec_e = np.array(lines, dtype=np.float64)
    src.spec_cdf = np.cumsum(yields) / np.sum(yields)
    scene = Scene(pt, _anatomy(labels, seed), [case["spacing"]] * 3, _corner(case), [WORLD] * 3, 0, src)
    size = case["pixels"]
    # the heads keep clear of the image: its corners lie inside the circle of rotation
    radius = max(250.0, 0.5 * math.hypot(case["nx"], case["ny"]) * case["spacing"] + 5.0)
    sp = S.SpectSpec(collimator=S.LEHR if case["nuclide"] == "tc99m" else S.MELP, n_runs=case["runs"],
                     windows=TC99M_WINDOWS if case["nuclide"] == "tc99m" else LU177_WINDOWS, radius=radius,
                     step_angle_deg=360.0 / case["runs"], collimator_material=n_ct, crystal_material=n_ct + 1,
                     size=(size, size), spacing=(565.76 / size,) * 2)
    sp.apply_housing(HOUSING, lambda m: n_ct + 2 + S.HOUSING_MATERIALS[HOUSING].index(m))
    return scene, sp


def _pinned(shape):
    """A float64 array in page-locked memory, as a program that fetches images again and again keeps."""
    return torch.empty(tuple(shape), dtype=torch.float64, pin_memory=True).numpy()


# ---- the ARF network --------------------------------------------------------------------
def _network(seed, n_classes, distance):
    """(model, parameters) of a network with He-uniform weights and small biases."""
    rng = np.random.default_rng([seed, 77])
    parts = []
    for fan, rows in ((3, HID), (HID, HID), (HID, HID), (HID, OUT_PAD)):
        parts.append(rng.uniform(-1, 1, (rows, fan)) * math.sqrt(6.0 / fan))
        parts.append(rng.uniform(-0.1, 0.1, rows))
    model = C.ArfModel()
    model.n_classes = n_classes
    model.x_mean[:] = [0.5 * THETA_MAX, 0.0, 0.5 * sum(E_RANGE)]
    model.x_std[:] = [THETA_MAX / math.sqrt(12), 360 / math.sqrt(12), (E_RANGE[1] - E_RANGE[0]) / math.sqrt(12)]
    model.russian_roulette = ROULETTE
    model.e_min, model.e_max = E_RANGE
    model.theta_max_deg = THETA_MAX
    model.distance_to_crystal = distance
    return model, np.concatenate([p.ravel() for p in parts]).astype(np.float32)


def _rows(seed, n):
    """Rows (E MeV, theta, phi deg, class) over the domain: the photopeak class near normal incidence at the
    line's energy, the scatter classes below, none at large angles."""
    rng = np.random.default_rng([seed, 5])
    r = np.empty((n, 4), dtype=np.float32)
    r[:, 0] = rng.uniform(*E_RANGE, n)
    r[:, 1] = rng.uniform(0.0, THETA_MAX, n)
    r[:, 2] = rng.uniform(-180.0, 180.0, n)
    seen = rng.uniform(size=n) < np.exp(-r[:, 1] / 12.0) + 0.15
    r[:, 3] = np.where(seen, 1 + np.digitize(-r[:, 0], [-0.1872, -0.166]), 0)
    return r


HEAD_MATERIALS = ("G4_AIR", "G4_Pb", "G4_SODIUM_IODIDE", *S.HOUSING_MATERIALS[HOUSING])


@functools.lru_cache(maxsize=None)
def _head_tables():
    db = M.MaterialDatabase()
    return T.PhysicsTables([db.get(n) for n in HEAD_MATERIALS])


def _head_engine(collimator):
    """An engine that holds only a head, as the ARF training step makes it."""
    src = SourceSpec()
    src.mono = 0.1
    scene = Scene(_head_tables(), np.zeros((1, 1, 1), np.uint16), [1.0] * 3, [-0.5] * 3, [2000.0] * 3, 0, src)
    sp = S.SpectSpec(collimator=S.COLLIMATORS[collimator], n_heads=1, n_runs=1, windows=LU177_WINDOWS,
                     collimator_material=1, crystal_material=2)
    sp.apply_housing(HOUSING, HEAD_MATERIALS.index)
    return SpectEngine(scene, sp)


# ---- prepare ----------------------------------------------------------------------------
def prepare(case, seed):
    seed = int(seed)
    return dict(case=case, seed=1000 + seed, **globals()["_prepare_" + case["kind"]](case, seed))


def _prepare_dose(case, seed):
    scene = _dose_scene(case, seed)
    eng = DoseEngine(scene, precision=case["precision"])
    which = [C.GG_IMG_EDEP, C.GG_IMG_EDEP_SQUARED]
    if case["grid"]:
        # voxels `grid` times as large, one and a half voxels beyond the image's corner, a little smaller than it
        f, dims = case["grid"], scene.dims_xyz
        step = [f * v for v in scene.spacing]
        eng.set_dose_grid([max(1, d // f - 1) for d in dims], step,
                          [c - 1.5 * s for c, s in zip(scene.corner, scene.spacing)])
        which += [C.GG_IMG_DOSE, C.GG_IMG_DOSE_SQUARED]
    if case["tle"]:
        eng.set_tle()
    return dict(eng=eng, images={w: _pinned(eng.image_shape()) for w in which})


def _prepare_batched(case, seed):
    rng = np.random.default_rng([seed, 3])
    # the sizes of the simulations are the case's, their contents the seed's
    sims = [(_slab_scene(rng, side), n, seed * 1000 + k) for k, (side, n) in enumerate(_batch_sizes(case))]
    eng = BatchEngine(sims)
    eng.capture()
    return dict(eng=eng, images=[(k, w, _pinned(s.labels.shape)) for k, (s, _, _) in enumerate(sims)
                                 for w in (C.GG_IMG_EDEP, C.GG_IMG_EDEP_SQUARED)])


def _batch_sizes(case):
    """(voxels a side, primaries) of each simulation of a batched case."""
    rng = np.random.default_rng(case["sims"])
    lo, hi = math.log(case["primaries_lo"]), math.log(case["primaries_hi"])
    return [(int(rng.choice((32, 48, 64, 96, 128))), int(math.exp(rng.uniform(lo, hi)))) for _ in range(case["sims"])]


def _slab_scene(rng, side):
    """A cube of `side` voxels in one to four slabs, a monoenergetic disc beam on its entrance face."""
    vm, lut, pt, _ = _ct_materials(False)
    hu = rng.choice(W.SLAB_HU, int(rng.integers(1, 5)))
    column = M.create_label_image(hu.astype(np.int16)[:, None, None], "G4_AIR", vm, lut)[:, 0, 0]
    labels = np.repeat(column[np.sort(rng.integers(0, len(hu), side))], side * side).reshape(side, side, side)
    spacing = float(rng.uniform(1.0, 3.0))
    half, src = side * spacing / 2.0, SourceSpec()
    src.pos_type = C.GG_POS_DISC
    src.radius = 10.0
    src.translation = [0.0, 0.0, -half - 1.0]
    src.dir_type = C.GG_DIR_MOMENTUM
    src.momentum = [0.0, 0.0, 1.0]
    src.ene_type = C.GG_ENE_MONO
    src.mono = math.exp(rng.uniform(math.log(0.05), math.log(2.0)))
    return Scene(pt, labels, [spacing] * 3, [-half] * 3, [500.0] * 3, 0, src)


def _prepare_spect(case, seed):
    scene, sp = _spect_scene(case, seed)
    runs = case["runs"]
    per_run = max(8, case["primaries"] // runs)
    if case["recipe"] == "plain":
        eng = SpectEngine(scene, sp)
        return dict(eng=eng, per_run=per_run, counts=_pinned(sp.projection_shape()))
    ff = case["recipe"] == "ff"
    share, forced, cone = (4, 1 / 8, 20.0) if ff else (8, 1 / 32, 10.0)
    prim, scat = copy.deepcopy(sp), copy.deepcopy(sp)
    prim.set_free_flight(angle_tolerance_max=0.0 if ff else math.radians(cone))
    scat.set_scatter_splitting(*((50, 10) if ff else (10, 2)), 10000, angle_tolerance_max=math.radians(10.0))
    aimed = copy.copy(scene)
    src = copy.copy(scene.source)
    src.dir_type = C.GG_DIR_FORCED
    src.fd_angle_min, src.fd_angle_max = 0.0, math.radians(cone)
    aimed.set_source(src)
    engines = SpectEngine(aimed, prim), SpectEngine(scene, scat)
    if not ff:
        model, params = _network(seed, sp.n_windows + 1, sp.crystal_depth())
        for e in engines:
            ArfNetwork(e).set_model(model, params)
            e.use_arf(True)
    return dict(prim=engines[0], scat=engines[1], per_prim=max(N_HEADS, int(round(per_run * forced)) * N_HEADS),
                per_scat=max(1, per_run // share))


def _prepare_arf_dataset(case, seed):
    eng = _head_engine(case["collimator"])
    smp = ArfNetwork.sampling(*E_RANGE, THETA_MAX, (200.0, 200.0), 1.0)
    return dict(net=ArfNetwork(eng), sampling=smp)


def _prepare_arf_train(case, seed):
    return dict(net=ArfNetwork(_head_engine("melp")), rows=_rows(seed, case["rows"]))


def _prepare_arf_predict(case, seed):
    net = ArfNetwork(_head_engine("melp"))
    net.set_model(*_network(seed, len(LU177_WINDOWS) + 1, 47.0))
    return dict(net=net, rows=_rows(seed, case["rows"]))


# ---- run --------------------------------------------------------------------------------
def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def _run_dose(s):
    eng = s["eng"]
    eng.reset()
    eng.run(s["case"]["primaries"], s["seed"])
    return dict(images={str(w): eng.image(w, out) for w, out in s["images"].items()}, counters=eng.counters())


def _run_batched(s):
    eng = s["eng"]
    eng.reset()
    eng.replay()
    return [eng.image(k, w, out) for k, w, out in s["images"]]


def _run_spect(s):
    if "eng" in s:
        eng = s["eng"]
        eng.reset()
        eng.run(s["per_run"], s["seed"])
        return dict(counts=eng.projection(s["counts"]), counters=eng.counters())
    out = {}
    for name, per in (("prim", "per_prim"), ("scat", "per_scat")):
        eng = s[name]
        eng.reset()
        eng.run(s[per], s["seed"])
        out[name], out[name + "_squared"] = eng.weighted_projection(squared=True)
        out[name + "_counters"] = eng.counters()
        if s["case"]["recipe"] == "arf":
            out[name + "_tracked"] = eng.projection()  # photons outside the network's domain
    return out


def _run_arf_dataset(s):
    return s["net"].dataset(s["sampling"], s["case"]["samples"], s["seed"])


def _run_arf_train(s):
    c = s["case"]
    _, loss = s["net"].train_rows(s["rows"], *E_RANGE, THETA_MAX, ROULETTE, epochs=c["epochs"], batch=c["batch"],
                                  lr=2e-3, lr_final=1e-5, init_seed=s["seed"])
    return dict(params=s["net"].params(), loss=loss)


def _run_arf_predict(s):
    return s["net"].predict(s["rows"])


# ---- work -------------------------------------------------------------------------------
# Arithmetic that a history cannot do without, from the mean number of flights, collisions and crossed voxels
# per primary of these phantoms (counters of the runs): a flight (path length, move, voxel, attenuation, test)
# is about 60 operations, a collision with its new direction and path to the boundary about 200, the source
# about 100, a voxel crossed by a straight path about 15.
def _history_flops(flights, collisions, crossed=0):
    return 100 + 60 * flights + 200 * collisions + 15 * crossed


def work(case):
    kind = case["kind"]
    if kind == "dose":
        vox = case["nx"] * case["ny"] * case["nz"]
        tallied = vox / case["grid"] ** 3 * 2 if case["grid"] else vox
        return dict(bytes=2 * vox + 16 * tallied,
                    flops=case["primaries"] * _history_flops(3.8, 1.6, 60 if case["tle"] else 0))
    if kind == "batched":
        sizes = _batch_sizes(case)
        return dict(bytes=sum(18 * side ** 3 for side, _ in sizes),
                    flops=sum(n for _, n in sizes) * _history_flops(3.0, 1.6))
    if kind == "spect":
        windows = len(TC99M_WINDOWS if case["nuclide"] == "tc99m" else LU177_WINDOWS)
        pixels = N_HEADS * case["runs"] * windows * case["pixels"] ** 2
        scene = 6 * case["nx"] * case["ny"] * case["nz"]
        if case["recipe"] == "plain":
            return dict(bytes=scene + 8 * pixels, flops=case["primaries"] * _history_flops(8.0, 3.0))
        ff = case["recipe"] == "ff"
        forced, share, copies = (1 / 4, 1 / 4, 45) if ff else (1 / 16, 1 / 8, 9)
        flops = case["primaries"] * (forced * _history_flops(0, 0, 100) +
                                     share * (_history_flops(8.0, 3.0) + 3.0 * copies * 60))
        if not ff:
            flops += case["primaries"] * forced * _network_flops()
        return dict(bytes=2 * scene + 32 * pixels + (0 if ff else 16 * pixels), flops=flops)
    if kind == "arf_dataset":
        return dict(bytes=16 * case["samples"], flops=case["samples"] * _history_flops(8, 1))
    if kind == "arf_train":
        steps = -(-case["rows"] // case["batch"]) * case["epochs"]
        return dict(bytes=16 * case["rows"] + 4 * N_PARAMS, flops=3 * steps * case["batch"] * _network_flops())
    return dict(bytes=(16 + 4 * (len(LU177_WINDOWS) + 1)) * case["rows"], flops=case["rows"] * _network_flops())


def _network_flops():
    return 2 * (3 * HID + 2 * HID * HID + HID * OUT_PAD)


# ---- exact ------------------------------------------------------------------------------
def exact(case, seed):
    """The network's answers in 64 bits.  A Monte Carlo tally has no such value: its histories are decided by
    their working precision."""
    seed = int(seed)
    if case["kind"] == "arf_predict" and case["rows"] <= 2_000_000:
        _, params = _network(seed, len(LU177_WINDOWS) + 1, 47.0)
        rows = torch.from_numpy(_rows(seed, case["rows"])).double()
        net = _split(torch.from_numpy(params).double())
        return torch.cat([_probabilities(net, r, len(LU177_WINDOWS) + 1) for r in rows.split(65536)]).numpy()
    if case["kind"] == "arf_train" and case["rows"] * case["epochs"] <= 600_000:
        return _exact_train(case, seed)
    return None


def _split(p):
    """The layers' (weight, bias) of a parameter vector."""
    out, at = [], 0
    for fan, rows in ((3, HID), (HID, HID), (HID, HID), (HID, OUT_PAD)):
        out.append((p[at:at + rows * fan].view(rows, fan), p[at + rows * fan:at + rows * (fan + 1)]))
        at += rows * (fan + 1)
    return out


def _logits(net, rows, n_classes):
    x = torch.stack([(rows[:, 1] - 0.5 * THETA_MAX) / (THETA_MAX / math.sqrt(12)), rows[:, 2] / (360 / math.sqrt(12)),
                     (rows[:, 0] - 0.5 * sum(E_RANGE)) / ((E_RANGE[1] - E_RANGE[0]) / math.sqrt(12))], 1)
    for w, b in net[:-1]:
        x = torch.relu(x @ w.T + b)
    return (x @ net[-1][0].T + net[-1][1])[:, :n_classes]


def _probabilities(net, rows, n_classes):
    return torch.softmax(_logits(net, rows, n_classes), 1)


def _initial(seed, n_classes):
    """He-uniform start of the training: splitmix64 draws, zero biases, unused outputs zero."""
    mask = (1 << 64) - 1
    state, p = seed & mask, np.zeros(N_PARAMS)

    def fill(at, n, fan):
        nonlocal state
        lim = math.sqrt(6.0 / fan)
        for i in range(n):
            state = (state + 0x9E3779B97F4A7C15) & mask
            z = ((state ^ (state >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            p[at + i] = np.float32((((z ^ (z >> 31)) >> 11) / 9007199254740992.0 * 2.0 - 1.0) * lim)

    fill(0, HID * 3, 3)
    at = HID * 4
    for _ in range(2):
        fill(at, HID * HID, HID)
        at += HID * (HID + 1)
    fill(at, n_classes * HID, HID)
    return torch.from_numpy(p)


def _exact_train(case, seed):
    n_classes, batch, n = len(LU177_WINDOWS) + 1, case["batch"], case["rows"]
    rows = torch.from_numpy(_rows(seed, n)).double()
    p = _initial(1000 + seed, n_classes).requires_grad_(True)
    m, v, loss, t = torch.zeros(N_PARAMS).double(), torch.zeros(N_PARAMS).double(), [], 0
    steps = -(-n // batch)
    decay = math.log(1e-5 / 2e-3) / (steps * case["epochs"])
    for _ in range(case["epochs"]):
        total = 0.0
        for _ in range(steps):
            at = (torch.arange(batch) + t * batch % n) % n
            r = rows[at]
            one = torch.nn.functional.cross_entropy(_logits(_split(p), r, n_classes), r[:, 3].long())
            g, = torch.autograd.grad(one, p)
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            lr = 2e-3 * math.exp(decay * t)
            t += 1
            with torch.no_grad():
                p -= lr * (m / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
            total += float(one.detach())
        loss.append(total / steps)
    return dict(params=p.detach().numpy(), loss=np.array(loss))
