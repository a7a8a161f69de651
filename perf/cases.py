"""What the SAL-gradient treecode is timed on: the work its users have it do,
through the public entry points of ``salgpu``.

Meshes are masked Fibonacci lattices (an ocean of quasi-uniform cells) or
lon-lat cells with a fixed land mask (the MOM6-style grid, whose spacing
shrinks toward the poles); sea-surface heights are sums of plane waves with a red
spectrum up to about degree 128, scaled to 1 m RMS.  Masks, areas and heights follow from the seed.
A case's ``kind`` says which entry points it goes through:

* ``solve``: ``Grid.solve`` on device-resident fields, in one of three forms:
  ``ref`` (FP64, the reference's arithmetic), ``accurate`` (FP64, Cartesian
  interpolation) and ``mixed`` (the batched tensor-core form);
* ``fast_sum``: the drop-in ``fast_sum`` on host arrays, as code.f90 calls it
  once per time step;
* ``mom6``: ``proxy_source_compute``, ``pc_compute`` and ``pp_compute`` on one
  grid with host arrays, as mom6_code.f90 calls them;
* ``host``: ``Grid.solve_host``, a batch of fields in and out of pinned host
  arrays;
* ``direct``: the FP64 direct sum at sampled targets, the accuracy check.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.abspath(os.getcwd()), "sal-fort_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import salgpu as S  # noqa: E402

THETA = 0.7
EARTH_RADIUS_M = 6371220.0
FORMS = {"ref": S.FORM_REF, "accurate": S.FORM_ACCURATE, "mixed": S.FORM_MIXED}


def listed():
    return [
        # The smallest call: a coarse mesh, one field, the reference's
        # arithmetic.  Launches and latency decide.
        dict(name="ref_3000", kind="solve", form="ref", cells=3000, leaf=20, degree=8, fields=1),
        # A coarse ocean model's mesh (about 40,962 cells before the land mask).
        dict(name="ref_28673", kind="solve", form="ref", cells=28673, leaf=100, degree=8, fields=1),
        # The reference's own mesh size, one field: its namelist run.
        dict(name="ref_2313486", kind="solve", form="ref", cells=2313486, leaf=200, degree=8, fields=1),
        # The FP64 form with the accurate interpolation at a higher degree.
        dict(name="accurate_163842", kind="solve", form="accurate", cells=163842, leaf=200, degree=10, fields=1),
        # Served meshes: a single-field request on the smallest one and a
        # batch of several requests on a middle one, with the server's settings.
        dict(name="mixed_40962_1f", kind="solve", form="mixed", cells=40962, leaf=200, degree=8, fields=1,
             block=64, f16=1, chain=64, cta_groups=1),
        dict(name="mixed_163842_13f", kind="solve", form="mixed", cells=163842, leaf=200, degree=8, fields=13,
             block=64, f16=1, chain=64, cta_groups=1),
        # A small ensemble on a grid made for at most 32 fields (32-field blocks).
        dict(name="mixed_163842_24f_block32", kind="solve", form="mixed", cells=163842, leaf=200, degree=8, fields=24,
             block=32, f16=0, chain=0, cta_groups=0),
        # The largest: 64 fields on the reference's mesh size, with the
        # settings the tuner picks there.
        dict(name="mixed_2313486_64f", kind="solve", form="mixed", cells=2313486, leaf=200, degree=8, fields=64,
             block=64, f16=1, chain=64, cta_groups=4, proxy_unit=324),
        # The MOM6-style path on the 0.25 degree lon-lat grid.
        dict(name="mom6_1440x720", kind="mom6", nlon=1440, nlat=720, leaf=200, degree=8, ref_compat=1),
        # A Fortran host's call of every time step: host arrays in and out.
        dict(name="fast_sum_163842", kind="fast_sum", cells=163842, leaf=200, degree=8),
        # The accuracy check: 10,000 sampled targets against every cell.
        dict(name="direct_10000x655362", kind="direct", cells=655362, targets=10000),
        # An ensemble held by a host program: copies in, batched solve, copies out.
        dict(name="host_655362_16f", kind="host", form="mixed", cells=655362, leaf=200, degree=8, fields=16,
             block=64, f16=1, chain=64, cta_groups=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: mesh sizes over their logarithm, odd
    ones among them; leaf sizes, degrees and field counts over what the
    configurations and the server use."""
    kind = rng.choice(["ref", "ref", "accurate", "mixed", "mixed", "mixed", "block32", "mom6", "fast_sum", "direct",
                       "host"])
    leaf = rng.choice([60, 100, 150, 200])
    if kind in ("ref", "accurate"):
        # smallest meshes have leaves to match
        cells = _log_int(rng, 2000, 1500000)
        return dict(kind="solve", form=kind, cells=cells, leaf=rng.choice([20, 40]) if cells < 10000 else leaf,
                    degree=rng.choice([6, 8, 8, 10]) if kind == "accurate" else rng.choice([6, 8, 8]), fields=1)
    if kind in ("mixed", "host"):
        cells = _log_int(rng, 10000, 1500000 if kind == "mixed" else 300000)
        return dict(kind="solve" if kind == "mixed" else "host", form="mixed", cells=cells, leaf=rng.choice([100, 150, 200]), degree=8,
                    fields=rng.randint(1, 64), block=64, f16=rng.choice([0, 1, 1]), chain=rng.choice([32, 64]),
                    cta_groups=rng.choice([1, 2, 4]))
    if kind == "block32":
        return dict(kind="solve", form="mixed", cells=_log_int(rng, 10000, 400000), leaf=rng.choice([100, 200]), degree=8,
                    fields=rng.randint(2, 32), block=32, f16=0, chain=0, cta_groups=0)
    if kind == "mom6":
        nlat = _log_int(rng, 120, 600)
        return dict(kind="mom6", nlon=2 * nlat + rng.choice([0, 1]), nlat=nlat, leaf=leaf, degree=rng.choice([6, 8]),
                    ref_compat=rng.choice([0, 1]))
    if kind == "fast_sum":
        return dict(kind="fast_sum", cells=_log_int(rng, 10000, 700000), leaf=leaf, degree=rng.choice([6, 8]))
    cells = _log_int(rng, 3000, 900000)
    return dict(kind="direct", cells=cells, targets=min(cells, _log_int(rng, 100, 10000)))


# ------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _waves(pts, rng, count, lo, hi, nfields):
    """nfields sums of `count` plane waves of wavenumbers lo..hi with
    amplitudes falling as 1 / (1 + k), at pts (N, 3): (nfields, N)."""
    k = lo * (hi / lo) ** rng.random(count)
    d = rng.standard_normal((count, 3))
    d *= (k / np.linalg.norm(d, axis=1))[:, None]
    ph = rng.uniform(0.0, 2.0 * math.pi, count)
    c = rng.standard_normal((nfields, count)) / (1.0 + k)
    dev = pts.device
    basis = torch.cos(torch.as_tensor(d, device=dev) @ pts.T + torch.as_tensor(ph, device=dev)[:, None])
    return torch.as_tensor(c, device=dev) @ basis


def _keep_largest(field, keep):
    """Indices, ascending, of the `keep` cells where the field is largest."""
    order = torch.sort(field, descending=True, stable=True).indices[:keep]
    return torch.sort(order).values


def _mesh(case, rng):
    """(points (N, 3) on the device, areas (N,) on the host) of the case's mesh."""
    dev = _device()
    if "nlon" in case:
        nlon, nlat = case["nlon"], case["nlat"]
        lon = (torch.arange(nlon, dtype=torch.float64, device=dev) + 0.5) * (2.0 * math.pi / nlon)
        edge = -0.5 * math.pi + torch.arange(nlat + 1, dtype=torch.float64, device=dev) * (math.pi / nlat)
        lat = (0.5 * (edge[1:] + edge[:-1]))[:, None].expand(nlat, nlon)
        lon = lon[None, :].expand(nlat, nlon)
        pts = torch.stack([torch.cos(lat) * torch.cos(lon), torch.cos(lat) * torch.sin(lon), torch.sin(lat)], -1)
        pts = pts.reshape(-1, 3)
        band = (2.0 * math.pi / nlon) * (torch.sin(edge[1:]) - torch.sin(edge[:-1]))
        area = band[:, None].expand(nlat, nlon).reshape(-1) * EARTH_RADIUS_M ** 2
        land = np.random.default_rng(nlon)
        idx = _keep_largest(_waves(pts, land, 24, 1.0, 12.0, 1)[0], int(round(0.7 * nlon * nlat)))
        return pts[idx].contiguous(), area[idx].cpu().numpy()
    n = case["cells"]
    nl = int(round(n / 0.7))
    i = torch.arange(nl, dtype=torch.float64, device=dev)
    z = 1.0 - (2.0 * i + 1.0) / nl
    r = torch.sqrt(torch.clamp(1.0 - z * z, min=0.0))
    phi = i * (math.pi * (3.0 - math.sqrt(5.0)))
    pts = torch.stack([r * torch.cos(phi), r * torch.sin(phi), z], 1)
    pts /= torch.linalg.vector_norm(pts, dim=1, keepdim=True)
    idx = _keep_largest(_waves(pts, rng, 24, 1.0, 8.0, 1)[0], n)
    area = 4.0 * math.pi * EARTH_RADIUS_M ** 2 / nl * (1.0 + 0.1 * rng.uniform(-1.0, 1.0, n))
    return pts[idx].contiguous(), area


def _inputs(case, seed):
    """Mesh and fields of a case: points (N, 3) and fields (F, N) on the
    device, coordinates and areas on the host."""
    rng = np.random.default_rng(seed)
    pts, area = _mesh(case, rng)
    h = _waves(pts, rng, 96, 1.0, 128.0, case.get("fields", 1))
    h /= torch.sqrt((h * h).mean(dim=1, keepdim=True))
    xyz = np.ascontiguousarray(pts.cpu().numpy().T)
    return pts, h, (xyz[0], xyz[1], xyz[2]), area


def _targets(case, seed):
    rng = np.random.default_rng(seed + 1)
    return np.sort(rng.choice(case["cells"], size=case["targets"], replace=False)).astype(np.int32)


def _tree_and_list(case, xyz):
    dev = 0 if torch.cuda.is_available() else None
    tree = S.tree_traverse(*xyz, len(xyz[0]), case["leaf"], device=dev)
    return tree, S.dual_tree_traversal(tree, THETA, case["leaf"], device=dev)


def prepare(case, seed):
    kind = case["kind"]
    pts, h, xyz, area = _inputs(case, seed)
    n = len(area)
    if kind == "direct":
        w = torch.as_tensor(area, device=pts.device) * h[0]
        c = pts.T.contiguous()
        return dict(kind=kind, x=c[0], y=c[1], z=c[2], w=w, targets=torch.as_tensor(_targets(case, seed), device=pts.device))
    if kind == "mom6":
        tree = S.tree_traverse(*xyz, n, case["leaf"])
        pc, pp = S.single_tree_traversal(tree, THETA, case["leaf"], *xyz)
        grid = S.mom6_grid(tree, pc, pp, *xyz, area, case["degree"], ref_compat=bool(case["ref_compat"]))
        return dict(kind=kind, grid=grid, h=h[0].cpu().numpy(), nw=(case["degree"] + 1) ** 2 * tree.npanels)
    tree, inter = _tree_and_list(case, xyz)
    if kind == "fast_sum":
        # the host program holds the flattened panels, as its own cube_panel array
        return dict(kind=kind, panels=tree.export(), inter=inter, xyz=xyz, area=area, h=h[0].cpu().numpy(),
                    degree=case["degree"])
    form = case["form"]
    grid = S.Grid(tree, *xyz, area, case["degree"], S.MODE_DTT, inter, max_fields=case.get("block", 1))
    if form == "mixed" and case["block"] == 64:
        more = {"proxy_unit_kpairs": case["proxy_unit"]} if "proxy_unit" in case else {}
        grid.tune(f16=case["f16"], chain_ksteps=case["chain"], cta_groups=case["cta_groups"], **more)
    if kind == "host":
        # pinned arrays, as numpy views of the tensors that own them
        keep = [torch.empty(h.shape, dtype=torch.float64, pin_memory=True) for _ in range(3)]
        keep[0].copy_(h)
        return dict(kind=kind, grid=grid, arrays=[k.numpy() for k in keep], keep=keep, form=FORMS[form])
    return dict(kind=kind, grid=grid, ssh=h, form=FORMS[form])


def _coords(case, seed):
    rng = np.random.default_rng(seed)
    pts, area = _mesh(case, rng)
    xyz = np.ascontiguousarray(pts.cpu().numpy().T)
    return pts, (xyz[0], xyz[1], xyz[2]), area


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "solve":
        return state["grid"].solve(state["ssh"], form=state["form"])
    if kind == "fast_sum":
        x, y, z = state["xyz"]
        gx, gy = np.zeros(len(x)), np.zeros(len(x))
        S.fast_sum(gx, gy, state["inter"], state["panels"], x, y, z, state["area"], state["h"], len(x), state["degree"],
                   with_points_inside=False)
        return gx, gy
    if kind == "mom6":
        g, h = state["grid"], state["h"]
        w, gx, gy = np.zeros(state["nw"]), np.zeros(len(h)), np.zeros(len(h))
        g.proxy_source_compute_host(h, w)
        g.pc_compute_host(w, gx, gy)
        g.pp_compute_host(h, gx, gy)
        return w, gx, gy
    if kind == "direct":
        return S.direct_sum(state["x"], state["y"], state["z"], state["w"], state["targets"])
    h, ox, oy = state["arrays"]
    state["grid"].solve_host(h, ox, oy, form=state["form"])
    return ox, oy


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Kernel pairs at 31 flops each and basis multiply-adds at 2 flops per
    component (FP64); in the batched form 4 flops per pair and field (two
    components, one multiply-add each) and the tree passes' multiply-adds.
    Bytes: coordinates, areas and fields in, results out."""
    kind = case["kind"]
    if kind == "direct":
        n, nt = case["cells"], case["targets"]
        return {"bytes": 32.0 * n + 20.0 * nt, "flops": 31.0 * n * nt}
    _, xyz, _ = _coords(case, 0)
    n = len(xyz[0])
    tree = S.tree_traverse(*xyz, n, case["leaf"])
    e = tree.export()
    count = np.diff(e["pt_off"]).astype(np.float64)
    P = (case["degree"] + 1) ** 2
    if kind == "mom6":
        pc, pp = S.single_tree_traversal(tree, THETA, case["leaf"], *xyz)
        pairs = float(len(pc)) * P + count[pp[:, 1] - 1].sum()
        return {"bytes": 56.0 * n + 8.0 * P * len(count), "flops": 31.0 * pairs + 2.0 * P * count.sum()}
    L = S.dual_tree_traversal(tree, THETA, case["leaf"])
    t, s, ty = L[:, 0] - 1, L[:, 1] - 1, L[:, 2]
    tcount = np.where((ty == 0) | (ty == 1), count[t], P)
    scount = np.where((ty == 0) | (ty == 2), count[s], P)
    pairs = (tcount * scount * (count[t] > 0) * (count[s] > 0)).sum()
    src = np.unique(s[(ty == 1) | (ty == 3)])
    tgt = np.unique(t[(ty == 2) | (ty == 3)])
    if case.get("form") == "mixed":
        F = case["fields"]
        return {"bytes": 32.0 * n + 24.0 * n * F, "flops": 4.0 * F * pairs + 8.0 * F * P * n}
    macs = P * (count[src].sum() + 2.0 * count[tgt].sum())
    return {"bytes": 56.0 * n, "flops": 31.0 * pairs + 2.0 * macs}


# ------------------------------------------------------------------ 64-bit values
def _direct_fields(pts, targets, weights):
    """Direct sums of sal_grad_gfunc over all sources for each field's
    weights (F, N), at target indices: two (F, T) tensors.  Elementwise
    operations in the kernel's own order, so that the self pair is the same
    rounding noise."""
    sx, sy, sz = (pts[:, k].contiguous() for k in range(3))
    F, T = weights.shape[0], len(targets)
    ox = torch.empty(F, T, dtype=torch.float64, device=pts.device)
    oy = torch.empty_like(ox)
    block = max(1, int(1.5e8 // len(sx)))
    wt = weights.T.contiguous()
    for b in range(0, T, block):
        t = pts[targets[b:b + block]]
        tx, ty, tz = t[:, 0:1], t[:, 1:2], t[:, 2:3]
        omz = 1.0 - tz * tz
        gxy = tx * sx
        gxy += ty * sy
        g = tz * sz
        g += gxy
        g.clamp_(-1.0, 1.0)
        mp = 2.0 - 2.0 * g
        q = torch.sqrt(mp)
        d2 = g * g
        d2 -= 1.0
        d2 *= 2.0
        d2 += 1e-16
        n2 = 2.0 * g
        n2 += q
        n2 *= 2.7 + 6.0
        n2 /= d2
        q *= mp
        q += 1e-16
        v = (1.0 - 6.21196) / q
        v += n2
        v *= -2.343256857908601e-9
        inv = torch.where((torch.abs(tz - 1.0) > 1e-15) & (torch.abs(tz + 1.0) > 1e-15), 1.0 / torch.sqrt(omz),
                          torch.zeros_like(omz))
        v *= inv
        k = sz * omz
        gxy *= tz
        k -= gxy
        k *= v
        oy[:, b:b + block] = (k @ wt).T
        k = tx * sy
        k -= ty * sx
        k *= v
        ox[:, b:b + block] = (k @ wt).T
    return ox, oy


def exact(case, seed):
    """The FP64 direct sum the treecode approximates, where it takes a few
    seconds at most (the proxy weights have no such value)."""
    kind = case["kind"]
    if kind == "direct":
        pts, h, _, area = _inputs(case, seed)
        tg = torch.as_tensor(_targets(case, seed).astype(np.int64), device=pts.device)
        ox, oy = _direct_fields(pts, tg, torch.as_tensor(area, device=pts.device) * h)
        return ox[0], oy[0]
    n = case["cells"] if "cells" in case else int(round(0.7 * case["nlon"] * case["nlat"]))
    if n > 200000:
        return None
    pts, h, _, area = _inputs(case, seed)
    ox, oy = _direct_fields(pts, torch.arange(n, device=pts.device), torch.as_tensor(area, device=pts.device) * h)
    if kind == "fast_sum":
        return ox[0], oy[0]
    if kind == "mom6":
        return None, ox[0], oy[0]
    return ox, oy
