"""The performance cases: the calls a user of this framework makes, over the range they are made in.

A case is one call (with its read-back) on a handle that the user's program keeps. `family` says through which
entry point it goes:

* semi       a semi-infinite medium: Engine(SIM_MCSUB), reset + run + results + summary
* voxel      a voxel tissue map: Engine(SIM_MCXYZ / SIM_MCXYZ_TT), the same calls
* sweep      many parameter sets in one launch: Engine.run_sweep / Engine.run_sweep_tissues
* layered    a stack of plane layers: layered.run, or layered.adjoint for per-layer gradients
* gradient   per-voxel media with a loss on Rd(r) or on Rd(r) and the fluence: autograd.transport, forward + backward
* field      polarised E-field transport with the coherent-backscattering cone, maps and Raman: efield.run
* speckle    mutual interference of recorded speckles: efield.speckle_mutual

`photons` is the whole call's number. Random walks have no closed form in 64 bits, so only `speckle` has exact values.
"""
import math

import numpy as np
import torch

from nmc_gb300 import abi, autograd, efield, engine, layered

AIR, EPIDERMIS, DERMIS, BLOOD = 1, 2, 3, 4
TWO_TERM = dict(gf=0.9, af=0.5, gb=0.3, ab=0.5, cc=0.9)  # forward and backward lobe, mean cosine 0.78


def listed():
    return [
        # one dispatch of the semi-infinite kernel: the smallest call, as a fit of a measured Rd(r) makes it again and again
        dict(name="semi_dispatch", family="semi", phase="hg", stream="philox", beam=0, mua=1.0, mus=100.0, g=0.9, bins=101, dr=0.002,
             photons=10_000),
        # the benchmark's semi-infinite medium at its launch size, with F(r, z)
        dict(name="semi_million", family="semi", phase="hg", stream="philox", beam=0, mua=1.0, mus=100.0, g=0.9, bins=101, dr=0.01,
             photons=1_000_000),
        # a 351-wavelength spectrum of the semi-infinite medium at pilot budgets, two-term phase function
        dict(name="semi_spectrum", family="sweep", geometry="semi", phase="tt", sets=351, photons=3_510_000),
        # what the nmc program runs by default: 1e5 photons on the reference's own streams through the skin-vessel map
        dict(name="vessel_program", family="voxel", scene="vessel", kernel="hg", stream="reference", source="uniform", boundary=2, det=0,
             nx=200, ny=200, nz=200, d=0.005, photons=100_000),
        # a converged fluence map of the same tissue, the benchmark's headline workload
        dict(name="vessel_fluence", family="voxel", scene="vessel", kernel="hg", stream="philox", source="uniform", boundary=2, det=0,
             nx=200, ny=200, nz=200, d=0.005, photons=10_000_000),
        # the two-term kernel on an odd, non-cubic grid with an inclusion, photons killed at the grid's faces
        dict(name="inclusion_two_term", family="voxel", scene="inclusion", kernel="tt", stream="philox", source="uniform", boundary=1, det=0,
             nx=41, ny=37, nz=29, d=0.011, photons=300_000),
        # a focused Gaussian beam through a thin odd slab, detected in transmittance
        dict(name="slab_transmittance", family="voxel", scene="slab", kernel="hg", stream="philox", source="gaussian", boundary=1, det=1,
             nx=97, ny=75, nz=16, d=0.01, photons=1_000_000),
        # a 351-wavelength spectrum of the skin-vessel map at pilot budgets, two-term phase function
        dict(name="vessel_spectrum", family="sweep", geometry="vessel", phase="tt", sets=351, photons=3_510_000),
        # three-layer skin: Rd(r), Tt(r), A(z)
        dict(name="skin_layers", family="layered", layers=3, nr=100, nz=100, a_rz=False, gradient=False, photons=1_000_000),
        # an inverse problem's step: gradients of Rd(r) and of the fluence for every voxel's mua, mus, g
        dict(name="voxel_gradient", family="gradient", n=64, d=0.01, bins=128, loss="both", photons=1_000_000),
        # the backscattering cone of a suspension: eight polarisation and incidence settings, Raman, maps
        dict(name="suspension_cone", family="field", settings=8, raman=True, cone_n=256, map_n=64, photons=1_000_000),
        # speckle post-processing of an exit map
        dict(name="speckle_map", family="speckle", nx=256, ny=256, records=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(("semi", "voxel", "voxel", "sweep", "layered", "gradient", "field", "speckle"))
    if family == "semi":
        case = dict(family=family, phase=rng.choice(("hg", "hg", "isotropic", "tt")), stream=rng.choice(("philox", "reference")),
                    beam=rng.choice((0, 0, 1, 2)), mua=round(rng.uniform(0.2, 5.0), 3), mus=round(rng.uniform(20.0, 300.0), 2),
                    g=round(rng.uniform(0.0, 0.95), 3), bins=rng.choice((51, 100, 101, 128, 200)), dr=rng.choice((0.002, 0.01)),
                    photons=_log(rng, 3_000, 5_000_000))
    elif family == "voxel":
        scene = rng.choice(("vessel", "inclusion", "slab", "cube"))
        kernel = rng.choice(("hg", "hg", "tt"))
        nx = _log(rng, 30, 200)
        case = dict(family=family, scene=scene, kernel=kernel, stream=rng.choice(("philox", "reference")),
                    source=rng.choice(("uniform", "isotropic", "square", "point", "pencil") + (("gaussian",) if kernel == "hg" else ())),
                    boundary=rng.choice((0, 1, 2)), det=1 if scene == "slab" and kernel == "hg" else 0, nx=nx,
                    ny=max(20, nx - rng.randint(0, 20)), nz=rng.randint(12, 40) if scene == "slab" else max(30, nx - rng.randint(0, 30)),
                    d=round(rng.uniform(0.005, 0.02), 4), photons=_log(rng, 3_000, 5_000_000))
    elif family == "sweep":
        sets = _log(rng, 8, 1000)
        case = dict(family=family, geometry=rng.choice(("semi", "vessel")), phase=rng.choice(("hg", "tt")), sets=sets,
                    photons=sets * _log(rng, 1_000, 20_000))
    elif family == "layered":
        case = dict(family=family, layers=rng.randint(1, 6), nr=rng.randint(50, 400), nz=rng.randint(50, 400), a_rz=rng.random() < 0.4,
                    gradient=rng.random() < 0.3, photons=_log(rng, 3_000, 3_000_000))
    elif family == "gradient":
        case = dict(family=family, n=_log(rng, 24, 80), d=0.01, bins=rng.choice((50, 128, 200)), loss=rng.choice(("rd", "both")),
                    photons=_log(rng, 10_000, 2_000_000))
    elif family == "field":
        settings = rng.randint(1, 12)
        case = dict(family=family, settings=settings, raman=rng.random() < 0.5, cone_n=rng.choice((64, 128, 256)),
                    map_n=rng.choice((32, 64, 100)), photons=settings * _log(rng, 2_000, 100_000))
    else:
        case = dict(family=family, nx=_log(rng, 60, 256), ny=_log(rng, 60, 256), records=_log(rng, 4, 64))
    if "photons" in case:  # a drawn case costs no more than the largest listed one
        case["photons"] = max(1, min(case["photons"], int(1e12 / (_steps(case) * _FLOPS[family]))))
    return case


# ---------------------------------------------------------------- work
_FLOPS = dict(semi=164, voxel=64, sweep=164, layered=170, gradient=192, field=320, speckle=250)  # lane operations per step (or record)


def _interactions(mua, mus):
    """Scatterings per photon of a thick medium, as the kernels count them (within a factor of two)."""
    return 31.0 * ((mua + mus) / mua) ** 0.56


def _steps(case):
    f = case["family"]
    if f == "semi":
        return _interactions(case["mua"], case["mus"])
    if f == "voxel":
        if case["scene"] == "vessel":
            return _interactions(0.5, 200.0) * (1 + 1.5 / (200.0 * case["d"]))
        if case["scene"] == "slab" or case["boundary"] == 1:  # most photons leave such a grid early
            return min(1.6 * 80.0 * min(case["nx"], case["ny"], case["nz"]) * case["d"], 300.0) * (1 + 1.5 / (80.0 * case["d"]))
        return _interactions(1.0, 100.0) * (1 + 1.5 / (100.0 * case["d"]))
    if f == "sweep":
        return _interactions(1.0, 100.0) if case["geometry"] == "semi" else 2.5 * _interactions(2.0, 100.0)
    if f == "layered":
        return _interactions(0.15, 120.0)
    if f == "gradient":
        return 300.0
    if f == "field":
        return _interactions(0.01, 100.0)
    return 1.0


def work(case):
    f = case["family"]
    if f == "speckle":
        pix = case["nx"] * case["ny"]
        return {"bytes": pix * (28.0 * case["records"] + 4 + 3 * 40), "flops": _FLOPS[f] * pix * float(case["records"])}
    if f == "voxel":
        byts = 5.0 * case["nx"] * case["ny"] * case["nz"] + 8.0 * case["nx"] * case["ny"] + 4.0 * abi.PHOTON_BATCH_DEFAULT
    elif f == "semi":
        byts = 4.0 * (case["bins"] + 1) * (case["bins"] + 2)
    elif f == "sweep":
        byts = case["sets"] * 200.0
    elif f == "layered":
        byts = 8.0 * (2 * case["nr"] + case["nz"] + (case["nr"] * case["nz"] if case["a_rz"] else 0))
    elif f == "gradient":
        byts = case["n"] ** 3 * (3 * 4 + 4 + 3 * 4.0)
    else:
        byts = case["settings"] * (16.0 * case["cone_n"] ** 2 + 40.0 * case["map_n"] ** 2)
    return {"bytes": byts, "flops": _FLOPS[f] * _steps(case) * case["photons"]}


# ---------------------------------------------------------------- inputs
def _scene(case, r):
    """uint8 map [iz, ix, iy], the run parameters and the tissue table of a voxel case."""
    nx, ny, nz, d = case["nx"], case["ny"], case["nz"], case["d"]
    y = (np.arange(ny) + 0.5 - ny / 2) * d
    x = (np.arange(nx) + 0.5 - nx / 2) * d
    z = (np.arange(nz) + 0.5) * d
    zsurf, n1 = 2 * d, 1.37
    jitter = lambda v: [float(q * r.uniform(0.98, 1.02)) for q in v]  # noqa: E731
    if case["scene"] == "vessel":  # air, epidermis, dermis and a blood vessel along x
        T = np.full((nz, nx, ny), DERMIS, np.uint8)
        T[:2] = AIR
        T[2:2 + max(1, round(0.006 / d))] = EPIDERMIS
        depth = 0.05 + r.uniform(-0.002, 0.002)
        T[np.broadcast_to(((y[None, None, :] ** 2 + (z[:, None, None] - depth) ** 2) <= 0.01 ** 2), T.shape)] = BLOOD
        mua, mus, g = jitter([0.0001, 20.0, 0.5, 230.0]), jitter([1.0, 300.0, 200.0, 200.0]), [1.0, 0.9, 0.9, 0.9]
    elif case["scene"] == "inclusion":  # a sphere under the surface
        T = np.full((nz, nx, ny), 2, np.uint8)
        T[:2] = AIR
        T[(x[None, :, None] ** 2 + y[None, None, :] ** 2 + (z[:, None, None] - 0.1) ** 2) <= 0.06 ** 2] = 3
        mua, mus, g = jitter([0.0001, 1.0, 5.0]), jitter([1.0, 80.0, 120.0]), [1.0, 0.85, 0.9]
    elif case["scene"] == "slab":
        T = np.full((nz, nx, ny), 2, np.uint8)
        T[:2] = AIR
        mua, mus, g = jitter([0.0001, 1.0]), jitter([1.0, 80.0]), [1.0, 0.85]
    else:  # a homogeneous cube
        T, zsurf, n1 = np.ones((nz, nx, ny), np.uint8), 0.0, 1.4
        mua, mus, g = jitter([1.0]), jitter([100.0]), [0.9]
    two = {k: [v] * len(mua) for k, v in TWO_TERM.items()} if case["kernel"] == "tt" else {}
    tp = abi.tissue_params(mua=mua, mus=mus, g=g, **two)
    source = dict(uniform=dict(mcflag=0, radius=0.03, waist=0.03), gaussian=dict(mcflag=1, radius=0.02, waist=0.02, zfocus=0.1),
                  isotropic=dict(mcflag=2, zs=zsurf + 0.05), square=dict(mcflag=3, radius=0.05), point=dict(mcflag=4),
                  pencil=dict(launchflag=1, xs=0.01, ys=-0.02, ux0=0.3, uy0=0.2, uz0=math.sqrt(1 - 0.13)))[case["source"]]
    kind = abi.SIM_MCXYZ_TT if case["kernel"] == "tt" else abi.SIM_MCXYZ
    rp = dict(myname="case", Nx=nx, Ny=ny, Nz=nz, dx=d, dy=d, dz=d, mcflag=0, launchflag=0, boundaryflag=case["boundary"], xs=0.0, ys=0.0,
              zs=zsurf + 1e-4, xfocus=0.0, yfocus=0.0, zfocus=float("inf"), ux0=0.0, uy0=0.0, uz0=1.0, radius=0.0, waist=0.0, zsurf=zsurf,
              det_radius=15.0, xd=0.0, n1=n1, n2=1.0, na=90.0, det_state=case["det"], mckernelflag=kind, Nt=len(mua))
    if case["det"]:
        rp["zsurf"] = nz * d
    return kind, abi.run_params(**{**rp, **source}), tp, T.reshape(-1)


def _smooth(shape, r, sigma):
    """White noise smoothed by a periodic Gaussian of `sigma` voxels, in [0, 1]."""
    k = [(2 * np.pi * np.fft.fftfreq(n)) ** 2 for n in shape]
    kk = k[0][:, None, None] + k[1][None, :, None] + k[2][None, None, :]
    s = np.real(np.fft.ifftn(np.fft.fftn(r.standard_normal(shape)) * np.exp(-0.5 * sigma ** 2 * kk)))
    return (s - s.min()) / (s.max() - s.min())


def _spectrum(r, n, lo, hi, base):
    """mua and mus of one tissue over n wavelengths: Gaussian absorption bands, power-law reduced scattering."""
    lam = np.linspace(400.0, 750.0, n)
    k = int(r.integers(3, 7))
    amp, cen, wid = r.uniform(lo, hi, k), r.uniform(400.0, 750.0, k), r.uniform(10.0, 60.0, k)
    mua = base + (amp * np.exp(-((lam[:, None] - cen) ** 2) / (2 * wid ** 2))).sum(1)
    return mua, r.uniform(10.0, 40.0) * (lam / 500.0) ** -r.uniform(0.8, 2.0) / (1 - 0.78)


def prepare(case, seed):
    r = np.random.default_rng(seed)
    f = case["family"]
    s = dict(case=case)
    if f == "semi":
        ref = case["stream"] == "reference"
        phase = dict(hg=abi.PHASE_HG, isotropic=abi.PHASE_ISOTROPIC_REF, tt=abi.PHASE_TWO_TERM)[case["phase"]]
        ext = abi.ext_defaults(rng=abi.RNG_TAUS_REF if ref else abi.RNG_PHILOX, seed=seed, phase=phase, sub_bins=case["bins"],
                               sub_dr=case["dr"], sub_dz=case["dr"], sub_mcflag=case["beam"], sub_radius=0.05 if case["beam"] else 0.0,
                               sub_zs=0.02 if case["beam"] == 2 else 0.0)
        jit = r.uniform(0.98, 1.02, 2)
        tp = abi.tissue_params(mua=[case["mua"] * jit[0]], mus=[case["mus"] * jit[1]], g=[case["g"]],
                               **({k: [v] for k, v in TWO_TERM.items()} if case["phase"] == "tt" else {}))
        rp = abi.run_params(myname="case", n1=1.37, n2=1.0, mckernelflag=abi.SIM_MCSUB, Nt=1)
        s["engine"] = engine.Engine(abi.SIM_MCSUB, 0, ext)
        s["engine"].prepare_data(rp, tp)
        s["first"] = (seed % 991) * ext.photons_per_dispatch if ref else 0
    elif f == "voxel":
        ref = case["stream"] == "reference"
        kind, rp, tp, v = _scene(case, r)
        ext = abi.ext_defaults(rng=abi.RNG_TAUS_REF if ref else abi.RNG_PHILOX, seed=seed)
        s["engine"] = engine.Engine(kind, 0, ext)
        s["engine"].prepare_data(rp, tp, v)
        s["first"] = (seed % 991) * ext.photons_per_dispatch if ref else 0
    elif f == "sweep":
        n, tt = case["sets"], case["phase"] == "tt"
        w = np.exp(r.uniform(0.0, math.log(10.0), n))  # uneven budgets, a factor of ten between the ends
        budgets = np.maximum(1, (w / w.sum() * case["photons"]).astype(np.int64))
        if case["geometry"] == "semi":
            mua, mus = _spectrum(r, n, 0.05, 2.0, 0.05)
            phase = abi.PHASE_TWO_TERM if tt else abi.PHASE_HG
            s["engine"] = engine.Engine(abi.SIM_MCSUB, 0, abi.ext_defaults(seed=seed, phase=phase))
            s["engine"].prepare_data(abi.run_params(myname="case", n1=1.37, n2=1.0, mckernelflag=abi.SIM_MCSUB, Nt=1),
                                     abi.tissue_params(mua=[1.0], mus=[100.0], g=[0.78], **{k: [v] for k, v in TWO_TERM.items()}))
            s["sets"] = [abi.SweepSet(mua=mua[i], mus=mus[i], g=0.78, n1=1.37, n2=1.0, pad=0, photons=int(budgets[i]), **TWO_TERM)
                         for i in range(n)]
        else:
            scene = dict(scene="vessel", kernel="tt" if tt else "hg", source="uniform", boundary=2, det=0, nx=200, ny=200, nz=200, d=0.005)
            kind, rp, tp, v = _scene(scene, r)
            s["engine"] = engine.Engine(kind, 0, abi.ext_defaults(seed=seed))
            s["engine"].prepare_data(rp, tp, v)
            bands = [_spectrum(r, n, lo, hi, 0.05) for lo, hi in ((1.0, 20.0), (0.05, 2.0), (10.0, 250.0))]
            s["tables"] = [abi.tissue_params(mua=[1e-4] + [b[0][i] for b in bands], mus=[1.0] + [b[1][i] for b in bands],
                                             g=[1.0, 0.78, 0.78, 0.78], **({k: [q] * 4 for k, q in TWO_TERM.items()} if tt else {}))
                           for i in range(n)]
            s["budgets"] = budgets
    elif f == "layered":
        skin = [(3.0, 200.0, 0.8, 1.4, 0.01), (0.3, 150.0, 0.85, 1.4, 0.2), (0.1, 100.0, 0.9, 1.44, 0.4), (1.0, 120.0, 0.9, 1.38, 0.1),
                (0.2, 80.0, 0.8, 1.42, 0.3), (0.5, 60.0, 0.9, 1.5, 0.5)][:case["layers"]]
        stack = [(a * r.uniform(0.95, 1.05), b * r.uniform(0.95, 1.05), g, n, t) for a, b, g, n, t in skin]
        s["stack"] = stack[:-1] + [stack[-1][:4] + (math.inf,)]
        s["kw"] = dict(nr=case["nr"], seed=seed)
        if case["gradient"]:
            s["up"] = dict(grad_rd_r=r.uniform(-1, 1, case["nr"] + 1).astype(np.float32),
                           grad_tt_r=r.uniform(-1, 1, case["nr"] + 1).astype(np.float32))
    elif f == "gradient":
        n, d = case["n"], case["d"]
        rp = abi.run_params(myname="case", Nx=n, Ny=n, Nz=n, dx=d, dy=d, dz=d, mcflag=0, launchflag=1, boundaryflag=1, xs=0.0, ys=0.0, zs=0.0,
                            xfocus=0.0, yfocus=0.0, zfocus=float("inf"), ux0=0.0, uy0=0.0, uz0=1.0, radius=0.0, waist=0.0, zsurf=0.0,
                            det_radius=15.0, xd=0.0, n1=1.4, n2=1.0, na=90.0, det_state=0, mckernelflag=abi.SIM_MCXYZ, Nt=1)
        e = s["engine"] = engine.Engine(abi.SIM_MCXYZ, 0, abi.ext_defaults(seed=seed))
        e.prepare_data(rp, abi.tissue_params(mua=[1.0], mus=[100.0], g=[0.85]), np.ones(n ** 3, np.uint8))
        e.set_radial_tally(case["bins"], 0.005)
        s["mua"] = torch.from_numpy((0.1 * 50.0 ** _smooth((n, n, n), r, 4.0)).astype(np.float32))
        s["mus"] = torch.from_numpy((50.0 + 250.0 * _smooth((n, n, n), r, 4.0)).astype(np.float32))
        s["g"] = torch.full((n, n, n), 0.85)
        s["up_rd"] = torch.from_numpy(r.uniform(0.5, 1.5, case["bins"] + 1).astype(np.float32))
        s["up_ab"] = torch.from_numpy(_smooth((n, n, n), r, 4.0).astype(np.float32)) if case["loss"] == "both" else None
    elif f == "field":
        rad = 0.5 * r.uniform(0.98, 1.02)  # spheres in water, um
        m = efield.sphere_suspension(rad, 1.59, 1.33, 633.0, 100.0)
        m700 = efield.mie(2 * math.pi * 1.33 * rad / 0.700, complex(1.59 / 1.33, 0.0), 1801)
        mus700 = m["number_density"] * m700["q_sca"] * math.pi * (rad * 1e-4) ** 2
        s["tables"] = (m["table"], m700["table"] if case["raman"] else None)
        s["config"] = abi.EfieldConfig(mua=0.01, mus=100.0, wavelength_cm=633e-7, raman_mua=0.01, raman_mus=mus700,
                                       raman_wavelength_cm=700e-7, mu_raman=1e-4 if case["raman"] else 0.0, n_medium=1.33, n_outside=1.0,
                                       n_angles=1801, cone_n=case["cone_n"], cone_half_angle=5e-3, sep_n=1024, sep_half_width=0.512,
                                       map_n=case["map_n"], map_dx=0.01, depth_bins=100, depth_dz=0.01, seed=seed, flags=0, speckle_max=0)
        s["settings"] = [abi.EfieldSetting(pol_angle=(k % 4) * math.pi / 4, theta_in=math.radians(10.0) * (k // 4 % 2), phi_in=0.0, pad=0,
                                           photons=case["photons"] // case["settings"]) for k in range(case["settings"])]
    else:
        nx, ny, k = case["nx"], case["ny"], case["records"]
        n = r.integers(max(1, k // 2), 2 * k + 1, (nx, ny))  # arrivals per pixel; the first `records` of them are kept
        maps = np.zeros((len(abi.EF_MAPS), nx, ny), np.float32)
        maps[abi.EF_MAPS.index("Det")] = n
        for q in ("XX", "XY", "YX", "YY", "Rd"):
            maps[abi.EF_MAPS.index(q)] = r.uniform(0, 1, (nx, ny)) * n
        for q in ("Phase0", "Phase1", "Phase2", "Phase3"):
            maps[abi.EF_MAPS.index(q)] = r.uniform(-math.pi, math.pi, (nx, ny)) * n
        rec = np.empty((k, nx, ny, 7), np.float32)
        rec[..., :4] = r.random((k, nx, ny, 4), np.float32) * np.float32(2 * math.pi) - np.float32(math.pi)
        rec[..., 4:] = r.random((k, nx, ny, 3), np.float32) * np.float32(0.2)
        s["maps"], s["counts"] = maps, np.minimum(n, k).astype(np.int32)
        s["records"] = rec.view(abi.SPECKLE_DTYPE)[..., 0]
    return s


# ---------------------------------------------------------------- the call
def run(state):
    case = state["case"]
    f = case["family"]
    if f in ("semi", "voxel"):
        e = state["engine"]
        e.reset()
        e.run(state["first"], case["photons"])
        out = e.get_compute_results()
        q = e.summary()
        out["sums"] = {k: q[k] for k in ("photons", "substeps", "scatters", "S", "A", "E", "rd_sum", "rd_sumsq")}
        return out
    if f == "sweep":
        e = state["engine"]
        if case["geometry"] == "semi":
            return e.run_sweep(state["sets"])
        return e.run_sweep_tissues(state["tables"], state["budgets"])
    if f == "layered":
        if case["gradient"]:
            return layered.adjoint(state["stack"], case["photons"], **state["up"], **state["kw"])
        return layered.run(state["stack"], case["photons"], nz=case["nz"], a_rz=case["a_rz"], **state["kw"])
    if f == "gradient":
        v = [state[k].clone().requires_grad_(True) for k in ("mua", "mus", "g")]
        if state["up_ab"] is None:
            rd = autograd.radial_reflectance(*v, state["engine"], n=case["photons"])
            rd.backward(state["up_rd"])
            return [rd.detach()] + [t.grad for t in v]
        rd, ab = autograd.transport(*v, state["engine"], n=case["photons"])
        ((rd * state["up_rd"]).sum() + (ab * state["up_ab"]).sum()).backward()
        return [rd.detach(), ab.detach()] + [t.grad for t in v]
    if f == "field":
        return efield.run(state["config"], state["tables"][0], state["settings"], state["tables"][1])
    return efield.speckle_mutual(state["maps"], state["records"], state["counts"], 633e-6, 0.05)


def exact(case, seed):
    if case["family"] != "speckle":
        return None
    s = prepare(case, seed)
    lam, lc, pi = 633e-6, 0.05, 3.1415926
    m = {k: s["maps"][i].astype(np.float64) for i, k in enumerate(abi.EF_MAPS)}
    wrap = lambda a: np.arctan2(np.sin(a), np.cos(a))  # noqa: E731
    norm = m["XX"] + m["XY"]
    xx, xy, rd, ph, pa, sc, tot = (m["XX"] / norm, m["XY"] / norm, *(m[k] / m["Det"] for k in ("Rd", "Phase0", "Phase1", "Phase2", "Phase3")))
    a = dict(XX=xx.copy(), XY=xy.copy(), Rd=rd.copy(), Phase0=ph.copy(), Phase1=pa.copy(), Phase2=sc.copy(), Phase3=tot.copy())
    for k in range(case["records"]):
        on = k < s["counts"]
        q = {n: s["records"][n][k].astype(np.float64) for n in abi.SPECKLE_DTYPE.names}
        both = q["XX"] + q["XY"]
        beat = np.sin(wrap(wrap(pa - q["Path"]) + wrap(sc - q["Scatt"])))
        beat = beat * np.exp(-(((q["Path"] - pa) * lam / (2 * pi)) / lc) ** 2)
        for n, u, v in (("XX", xx, q["XX"] / both), ("XY", xy, q["XY"] / both), ("Rd", rd, q["Ryx"])):
            a[n] += np.where(on, (u + v + 2 * np.sqrt(u * v) * beat) / 4, 0)
        for n, v in (("Phase0", q["Phase"]), ("Phase1", q["Path"]), ("Phase2", q["Scatt"]),
                     ("Phase3", wrap(q["Phase"] + q["Path"] + q["Scatt"]))):
            a[n] += np.where(on, v, 0)
    out = np.zeros(s["maps"].shape)
    for n, v in a.items():
        out[abi.EF_MAPS.index(n)] = v
    out[abi.EF_MAPS.index("Det")] = 1 + s["counts"]
    return out
