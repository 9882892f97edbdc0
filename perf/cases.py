"""Performance cases: the pair counts a user of this package runs, through its
public entry points, on seeded synthetic inputs (tos_b200.synth).

Kinds of case:

* ``xi``        pair count of one resident catalogue (tos_xi_run), in any of the
                three binnings, with whole or masked forests;
* ``mocks``     many mock catalogues batched in one run (TOS_XI_PER_GROUP);
* ``jackknife`` every delete-one-region subsample in one pass, then the
                covariance of the subsamples;
* ``plates``    sightlines binned by BOSS plate, with the per-plate sums and
                their covariance (the reference's do_cov);
* ``catalog``   a new catalogue: host arrays to the device, distances from the
                wavelengths there, one pair count, the catalogue given back;
* ``brute``     all pairs of points (x, y, z, delta, w), on a grid or scattered.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "turbo-octo-spice_b200"))

import tos_b200 as T  # noqa: E402
from tos_b200 import synth  # noqa: E402

FIELDS = ("didj", "di", "dj", "wgt", "wi", "wj", "z", "num_pairs")
DENSITY = 16.0     # quasars per square degree (the survey and mock configurations)
OMEGA_M = 0.3
ORDER = 6          # HEALPix nside = 64 cells
EXACT_PAIRS = 2.5e9  # pairs up to which exact() takes seconds


def _xi(name, n, coord, n0, n1, rmax, area=None, masked=0.0):
    c = {"kind": "xi", "n": n, "area": area or n / DENSITY, "coord": coord, "n0": n0, "n1": n1, "rmax": rmax,
         "masked": masked}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a few sightlines, where launches and copies count
        _xi("first_look_cart", 48, "cartesian", 50, 50, 200.0, area=9.0),
        # the small configuration: 2,000 quasars on 10 x 10 degrees, (r_par, r_perp) 50 x 50 to 200 Mpc/h
        _xi("patch_cart", 2000, "cartesian", 50, 50, 200.0, area=100.0),
        # a large piece of the survey at its density (the whole survey is ten times this)
        _xi("survey_cart", 16000, "cartesian", 50, 50, 200.0),
        # the same in (r, mu) 50 x 20
        _xi("survey_polar", 7000, "polar", 50, 20, 200.0),
        # real forests: sky lines, absorbers and bad pixels masked out, so pixels are not contiguous
        _xi("masked_cart", 1201, "cartesian", 50, 50, 200.0, masked=0.08),
        # observing coordinates (dloglam, theta): every pair of a patch
        _xi("patch_observing", 500, "observing", 25, 1, 0.05, area=100.0),
        # mock realisations of uneven size in one run
        {"name": "mock_batch", "kind": "mocks", "n": 5000, "mocks": 5, "n0": 50, "n1": 20, "rmax": 200.0},
        # jackknife subsamples of one mock, regions of HEALPix nside = 8
        {"name": "jackknife", "kind": "jackknife", "n": 2500, "region_order": 3, "n0": 50, "n1": 20, "rmax": 200.0},
        # BOSS plates with per-plate sums and their covariance
        {"name": "plates_cov", "kind": "plates", "n": 900, "area": 60.0, "n0": 50, "n1": 50, "rmax": 200.0},
        # a catalogue that is new to the device: upload, distances, one count, release
        {"name": "new_catalog", "kind": "catalog", "n": 3000, "area": 3000.0, "n0": 50, "n1": 50, "rmax": 200.0},
        # the brute-force configuration: 64^3 grid, 100 bins to 200 Mpc/h
        {"name": "brute_grid64", "kind": "brute", "grid": True, "n": 64 ** 3, "nbins": 100, "rmax": 200.0},
        # scattered points (pixels in space), where neighbouring pairs fall in unrelated bins
        {"name": "brute_points", "kind": "brute", "grid": False, "n": 20011, "nbins": 50, "rmax": 200.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["xi", "xi", "xi", "mocks", "jackknife", "plates", "catalog", "brute", "brute"])
    rmax = float(rng.choice([100, 140, 150, 180, 200]))
    cart = rng.choice([(50, 50), (40, 40), (28, 28), (47, 33), (20, 60)])
    pol = rng.choice([(50, 20), (25, 10), (41, 13), (50, 50)])
    if kind == "xi":
        coord = rng.choice(["cartesian", "cartesian", "polar", "observing"])
        if coord == "observing":
            return _xi(None, _log_int(rng, 40, 900), coord, rng.choice([13, 25, 50]), 1, rng.choice([0.03, 0.05]),
                       area=100.0, masked=rng.choice([0.0, 0.05]))
        masked = rng.choice([0.0, 0.0, 0.03, 0.1])
        n = _log_int(rng, 40, 1500 if masked else 7000)
        n0, n1 = cart if coord == "cartesian" else pol
        return _xi(None, n, coord, n0, n1, rmax, area=max(9.0, n / DENSITY), masked=masked)
    if kind == "mocks":
        k = rng.randint(2, 9)
        return {"kind": kind, "n": _log_int(rng, 100 * k, 6000), "mocks": k, "n0": pol[0], "n1": pol[1], "rmax": rmax}
    if kind == "jackknife":
        return {"kind": kind, "n": _log_int(rng, 400, 4000), "region_order": rng.choice([2, 3, 4]), "n0": pol[0],
                "n1": pol[1], "rmax": rmax}
    if kind == "plates":
        n = _log_int(rng, 80, 1500)
        return {"kind": kind, "n": n, "area": float(rng.choice([36, 60, 120])), "n0": cart[0], "n1": cart[1],
                "rmax": rmax}
    if kind == "catalog":
        n = _log_int(rng, 100, 6000)
        return {"kind": kind, "n": n, "area": n * rng.choice([0.5, 1.0, 2.0]), "n0": cart[0], "n1": cart[1],
                "rmax": rmax}
    grid = rng.random() < 0.5
    n = rng.randint(8, 60) ** 3 if grid else _log_int(rng, 500, 40000)
    return {"kind": kind, "grid": grid, "n": n, "nbins": rng.choice([20, 50, 100, 200]), "rmax": rmax}


def _grid(case):
    if case.get("coord") == "observing":
        return T.Grid.observing(dloglam="[0:%g]*%d" % (case["rmax"], case["n0"]))
    if case["kind"] in ("mocks", "jackknife") or case.get("coord") == "polar":
        return T.Grid.polar(r="[0:%g]*%d" % (case["rmax"], case["n0"]), mu="[0:1]*%d" % case["n1"])
    return T.Grid.cartesian(rpar="[0:%g]*%d" % (case["rmax"], case["n0"]),
                            rperp="[0:%g]*%d" % (case["rmax"], case["n1"]))


def _mask_pixels(los, px, fraction, seed):
    """Drop masked pixels: per forest three windows (sky lines, an absorber)
    and single bad pixels, about `fraction` of them in all."""
    rng = np.random.default_rng(seed)
    n = los["num_pixels"].astype(np.int64)
    first = los["pixel_offset"].astype(np.int64)
    keep = rng.random(len(px)) >= 0.2 * fraction
    for _ in range(3):
        width = np.maximum(1, (0.8 * fraction / 3 * n * rng.uniform(0.3, 1.7, len(n))).astype(np.int64))
        start = (rng.random(len(n)) * np.maximum(1, n - width)).astype(np.int64)
        cut = np.zeros(len(px) + 1, dtype=np.int32)
        np.add.at(cut, first + start, 1)
        np.add.at(cut, np.minimum(first + start + width, first + n), -1)
        keep &= np.cumsum(cut[:-1]) == 0
    total = np.concatenate([[0], np.cumsum(keep)])
    out = los.copy()
    out["pixel_offset"] = total[first]
    out["num_pixels"] = total[first + n] - total[first]
    return out, px[keep]


def _host(case, seed):
    """Host arrays of a case: (sightlines, pixels, scale, platelist or None), or the points of a brute case."""
    kind = case["kind"]
    if kind == "brute":
        rng = np.random.default_rng(seed)
        if case["grid"]:
            side = round(case["n"] ** (1.0 / 3.0))
            return synth.grf_grid(side, 4.0 * side, seed=seed)
        pts = np.empty((case["n"], 5), dtype=np.float32)
        pts[:, :3] = rng.uniform(0.0, 400.0, (case["n"], 3))
        pts[:, 3] = rng.normal(0.0, 0.2, case["n"])
        pts[:, 4] = rng.uniform(0.5, 2.0, case["n"])
        return pts
    if kind == "mocks":
        rng = np.random.default_rng(seed)
        share = np.exp(rng.uniform(-1.0, 1.0, case["mocks"]))
        counts = np.maximum(8, case["n"] * share / share.sum()).astype(int)
        parts, scale = [], math.inf
        for k, n in enumerate(counts):
            los, px, meta = synth.cap_patch(int(n), seed * 100 + k, n / DENSITY, omega_m=OMEGA_M)
            parts.append((los, px))
            scale = min(scale, meta["scale"])
        los, px = synth.merge_groups(parts)
        return los, px, scale, None
    if kind in ("jackknife", "plates"):
        # one footprint, so that every seed fills the same regions or plates; redshifts and pixels are the seed's
        side = math.sqrt(case.get("area", case["n"] / DENSITY))
        rng = np.random.default_rng(case["n"])
        ra = np.radians(rng.uniform(180.0, 180.0 + side, case["n"]))
        dec = np.arcsin(rng.uniform(math.sin(math.radians(20.0)), math.sin(math.radians(20.0 + side)), case["n"]))
        los, px, meta = synth.forest_catalog(ra, dec, seed, omega_m=OMEGA_M)
        if kind == "jackknife":
            return los, px, meta["scale"], None
        los, plates = synth.plate_tiling(los, 2.0)
        return los, px, meta["scale"], plates
    los, px, meta = synth.cap_patch(case["n"], seed, case["area"], omega_m=OMEGA_M)
    if case.get("masked"):
        los, px = _mask_pixels(los, px, case["masked"], seed + 1)
    return los, px, meta["scale"], None


def prepare(case, seed):
    """The engine, the grid and what the program holds before the call: the
    resident catalogue, or the host arrays where the call takes those."""
    s = {"kind": case["kind"], "case": case, "engine": T.Engine(0)}
    host = _host(case, seed)
    if case["kind"] == "brute":
        s["points"] = host
        return s
    los, px, s["scale"], plates = host
    s["grid"] = _grid(case)
    if case["kind"] == "catalog":
        s["los"], s["px"] = los, px
    elif case["kind"] == "plates":
        s["catalog"] = T.Catalog(s["engine"], los, px, platelist=plates)
    else:
        s["catalog"] = T.Catalog(s["engine"], los, px, ORDER)
    return s


def _columns(bins):
    return {f: bins[f] for f in FIELDS}


def run(s):
    eng, kind = s["engine"], s["kind"]
    if kind == "brute":
        dsum, wsum, counts, _ = T.brute_run(eng, s["points"], 0.0, s["case"]["rmax"], s["case"]["nbins"])
        return {"dsum": dsum, "wsum": wsum, "counts": counts.view(np.int64)}
    grid = s["grid"]
    if kind == "xi":
        return _columns(T.xi_run(eng, s["catalog"], grid, s["scale"])[0])
    if kind == "mocks":
        bins, rows, _ = T.xi_run(eng, s["catalog"], grid, s["scale"], per_group=True)
        return {"all": _columns(bins), "mocks": _columns(rows)}
    if kind == "jackknife":
        ids, bins, _, drop, _ = T.xi_run_jackknife(eng, s["catalog"], grid, s["scale"], s["case"]["region_order"])
        xi, mean, cov = T.subsample_covariance(eng, drop) if len(ids) > 1 else (drop["didj"], drop["wgt"], 0.0)
        return {"regions": ids, "all": _columns(bins), "drop": _columns(drop), "xi": xi, "mean": mean, "cov": cov}
    if kind == "plates":
        bins, rows, _ = T.xi_run(eng, s["catalog"], grid, s["scale"], subsamples=True)
        mean, cov, _ = T.cell_covariance(eng, s["catalog"], grid.nbins)
        return {"all": _columns(bins), "cells": _columns(rows), "mean": mean, "cov": cov}
    cat = T.Catalog(eng, s["los"], s["px"], ORDER, omega_matter=OMEGA_M)
    bins, _, _ = T.xi_run(eng, cat, grid, s["scale"])
    cat.close()
    return _columns(bins)


# A forest of this survey: 560 pixels in the mean, 3.35e5 in the mean square.
MEAN_PIXELS, MEAN_PIXELS2 = 560.0, 560.0 ** 2
# The transverse comoving distance at z = 1.96, the first pixel's (Mpc/h).
MEAN_SCALE = 3640.0


def _pixel_pairs(case):
    """Expected pixel pairs of the sightline pairs within the angular cut."""
    n = case["n"]
    if case.get("coord") == "observing":
        return 0.5 * n * (n - 1) * MEAN_PIXELS2
    cut = math.pi * (case["rmax"] / MEAN_SCALE * 180.0 / math.pi) ** 2  # square degrees
    if case["kind"] == "mocks":
        per = n / case["mocks"]
        return 1.25 * 0.5 * n * (per - 1) * min(1.0, cut * DENSITY / per) * MEAN_PIXELS2
    area = case.get("area", n / DENSITY)
    return 0.5 * n * (n - 1) * min(1.0, cut / area) * MEAN_PIXELS2 * (1.0 - case.get("masked", 0.0)) ** 2


def work(case):
    """Pixels (16 bytes) read once and bins (64 bytes) written once; two
    multiply-adds for every pair, its weight and its product of deltas."""
    if case["kind"] == "brute":
        n = case["n"]
        return {"bytes": 20.0 * n + 24.0 * (case["nbins"] + 2), "flops": 4.0 * 0.5 * n * (n - 1)}
    bins = case["n0"] * case["n1"]
    return {"bytes": 16.0 * MEAN_PIXELS * case["n"] + 64.0 * bins, "flops": 4.0 * _pixel_pairs(case)}


# ---- the same sums in 64 bits with plain torch --------------------------------

def _exact_brute(case, seed):
    pts = torch.from_numpy(_host(case, seed)).cuda().double()
    nb, rmax = case["nbins"], case["rmax"]
    spacing = (rmax - 0.0) / nb
    out = torch.zeros(2, nb + 2, dtype=torch.float64, device="cuda")
    n, wd = len(pts), pts[:, 4] * pts[:, 3]
    step = max(1, int(2e7 / n))
    for a in range(0, n, step):
        d = pts[a:a + step, None, :3] - pts[None, a:, :3]
        d2 = d * d
        r = torch.sqrt((d2[..., 0] + d2[..., 1]) + d2[..., 2])
        b = torch.clamp(torch.floor(r / spacing), 0, nb - 1).long() + 1
        b = torch.where(r >= rmax, nb + 1, b)
        i, j = torch.triu_indices(r.shape[0], r.shape[1], 1, device="cuda")
        k = b[i, j]
        out[0].index_add_(0, k, wd[a + i] * wd[a + j])
        out[1].index_add_(0, k, pts[a + i, 4] * pts[a + j, 4])
    return {"dsum": out[0].cpu().numpy(), "wsum": out[1].cpu().numpy(), "counts": None}


def _exact_xi(case, seed):
    los, px, scale, _ = _host(case, seed)
    grid = _grid(case)
    (a0, a1), nb = grid.axes[:2], grid.nbins
    coord = case["coord"]
    dev = {f: torch.from_numpy(px[f].copy()).cuda() for f in ("value", "loglam", "weight", "distance")}
    first, n = los["pixel_offset"].astype(np.int64), los["num_pixels"].astype(np.int64)
    sd, cd, sr, cr = np.sin(los["dec"]), np.cos(los["dec"]), np.sin(los["ra"]), np.cos(los["ra"])
    cos_max = math.cos(grid.max_angular_scale(scale))
    out = torch.zeros(7, nb + 1, dtype=torch.float64, device="cuda")  # the last column takes what is not binned

    def code(x, axis):  # the bin, or -1 outside (values in (-1, 0) bins fall into bin 0)
        t = (x - axis.min) * (1.0 / axis.width)
        k = torch.trunc(t).long()
        return torch.where((t > -1.0) & (k < axis.nbins), k, -1)

    owner = torch.from_numpy(np.repeat(np.arange(len(los)), n)).cuda()
    for i in range(len(los)):
        c = sd[i] * sd + cd[i] * cd * (cr[i] * cr + sr[i] * sr)
        ok = (c > cos_max) & (np.arange(len(los)) > i)
        if not ok.any():
            continue
        rows = slice(int(first[i]), int(first[i] + n[i]))
        cols = torch.nonzero(torch.from_numpy(ok).cuda()[owner]).flatten()
        cc = torch.from_numpy(c).cuda()[owner[cols]][None, :]
        l1, l2 = dev["loglam"][rows][:, None], dev["loglam"][cols][None, :]
        d1, d2 = dev["distance"][rows][:, None], dev["distance"][cols][None, :]
        if coord == "observing":
            k = code((l1 - l2).abs().double(), a0)  # theta (radians) lies in the one bin of its axis
        else:
            para = (d1 - d2).abs().double()
            sq = (d1 * d1).double() + (d2.double() - (2.0 * d1).double() * cc) * d2.double()
            if coord == "cartesian":
                k0, k1 = code(para, a0), code(torch.sqrt((sq - para * para).abs()), a1)
            else:
                r = torch.sqrt(sq)
                k0, k1 = code(r, a0), code(para / r, a1)
            k = torch.where((k0 >= 0) & (k1 >= 0), k1 + k0 * a1.nbins, -1)
        k = torch.where(k < 0, nb, k).flatten()
        w1, w2 = dev["weight"][rows].double()[:, None], dev["weight"][cols].double()[None, :]
        v1 = w1 * dev["value"][rows].double()[:, None]
        v2 = w2 * dev["value"][cols].double()[None, :]
        one = torch.ones_like(w1 * w2)
        for f, x in enumerate((v1 * v2, v1 * one, v2 * one, w1 * w2, w1 * one, w2 * one, 0.5 * (l1.double() + l2.double()))):
            out[f] += torch.bincount(k, weights=x.flatten(), minlength=nb + 1)
    res = {f: out[m, :nb].cpu().numpy() for m, f in enumerate(FIELDS[:7])}
    return dict(res, num_pairs=None)


def exact(case, seed):
    if case["kind"] == "brute":
        return _exact_brute(case, seed) if 0.5 * case["n"] ** 2 <= EXACT_PAIRS else None
    if case["kind"] == "xi" and _pixel_pairs(case) <= EXACT_PAIRS:
        return _exact_xi(case, seed)
    return None
