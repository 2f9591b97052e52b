"""The work that users of this package have it do, as cases that can be timed and compared.

A case is one call of a public entry point on inputs of a stated size and kind:
  mesh    extract_device: a volume resident on the GPU -> points, normals, triangles in device buffers that
          the caller keeps (float32 or integer samples; Flying Edges, Marching Cubes, duplicate-free order)
  batch   extract_batch_packed: many (volume, isovalue) requests in one call into reused buffers
  host    extract: a host volume in, a host mesh out -- the drop-in for the serial extraction call
  size    predictor.block_stats and Predictor.predict: mesh sizes from the output-size network
  train   predictor.mlp_gradient: one training step's gradients of that network
The fields are the two that the benchmark uses (sums of Gaussian blobs, octaves of value noise), drawn on
the GPU from the seed.
"""
import math
import random

import numpy as np
import torch

import miniisosurface_gb300 as M
from miniisosurface_gb300 import predictor as P

ALGOS = {"fe": M.FLYING_EDGES, "mc": M.MARCHING_CUBES, "dup": M.MC_DUPFREE}
MOST_POINTS = 768 ** 3  # of the largest listed volume


def mesh(name, algo, dims, field, iso, dtype="float32", index_bytes=4, unit=True):
    """unit False: spacing and origin that are no powers of two (the gradients divide by the spacing)."""
    return {"name": name, "kind": "mesh", "algo": algo, "nx": dims[0], "ny": dims[1], "nz": dims[2], "field": field,
            "iso": iso, "dtype": dtype, "index_bytes": index_bytes, "unit": unit}


def listed():
    return [
        # the smallest volume of the serving stream: launches and host latency are most of the call
        mesh("fe_64_blobs", "fe", (64, 64, 64), "blobs", 0.5),
        # the plain drop-in case: one small volume with a few closed surfaces
        mesh("fe_128_blobs", "fe", (128, 128, 128), "blobs", 0.5),
        # a cut-out of a scan: odd sizes, uneven spacing and origin, the reference's 64-bit indices
        mesh("fe_ragged_i64", "fe", (301, 217, 190), "noise", 0.1, index_bytes=8, unit=False),
        # the headline volume: one dense surface through 512^3 points
        mesh("fe_512_noise", "fe", (512, 512, 512), "noise", 0.0),
        # the largest volume of the serving stream, rows longer than 512 points
        mesh("fe_768_noise", "fe", (768, 768, 768), "noise", 0.0),
        # the headline volume through Marching Cubes
        mesh("mc_512_noise", "mc", (512, 512, 512), "noise", 0.0),
        # Marching Cubes on a simulation domain of uneven sides, rows longer than 512 points
        mesh("mc_667_blobs", "mc", (667, 228, 724), "blobs", 0.4, unit=False),
        # a scanner's 16-bit volume, extracted as it is
        mesh("fe_int16_512", "fe", (512, 512, 320), "noise", 0.0, dtype="int16"),
        # many small volumes of uneven sizes at several isovalues each, into one set of buffers
        {"name": "batch_64_volumes", "kind": "batch", "volumes": 64, "least": 32, "most": 320, "sizes": 2},
        # the serial call's own form: numpy volume in, numpy mesh out
        {"name": "host_256_noise", "kind": "host", "algo": "fe", "nx": 256, "ny": 256, "nz": 256, "field": "noise",
         "iso": 0.0},
        # admission of a new volume: its block statistics, then mesh sizes at four isovalues
        {"name": "size_320_noise", "kind": "size", "nx": 320, "ny": 320, "nz": 320, "isos": 4},
        # one step of training the output-size network at its batch size
        {"name": "train_16384", "kind": "train", "rows": 16384},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi, most):
    while True:
        d = [_spread(rng, lo, hi) for _ in range(3)]
        if d[0] * d[1] * d[2] <= most:
            return d


def draw(rng):
    kind = rng.choice(["mesh"] * 6 + ["batch", "host", "size", "train"])
    if kind == "batch":
        return {"kind": "batch", "volumes": _spread(rng, 4, 60), "least": 32, "most": rng.randint(96, 320),
                "sizes": rng.randint(10, 10 ** 6)}
    if kind == "train":
        return {"kind": "train", "rows": _spread(rng, 1000, 60000)}
    if kind == "size":
        d = _sides(rng, 64, 768, 320 ** 3)
        return {"kind": "size", "nx": d[0], "ny": d[1], "nz": d[2], "isos": rng.randint(1, 16)}
    field = rng.choice(["blobs", "noise"])
    iso = round(rng.uniform(0.3, 0.6) if field == "blobs" else rng.uniform(-0.4, 0.4), 3)
    if kind == "host":
        d = _sides(rng, 48, 320, 256 ** 3)
        return {"kind": "host", "algo": rng.choice(["fe", "fe", "mc"]), "nx": d[0], "ny": d[1], "nz": d[2],
                "field": field, "iso": iso}
    algo = rng.choice(["fe"] * 6 + ["mc"] * 3 + ["dup"])
    dtype = rng.choice(["float32"] * 6 + ["int16", "uint16", "uint8", "int8"])
    d = _sides(rng, 64, 768, MOST_POINTS // 2 if dtype == "float32" else 512 * 512 * 320)
    c = mesh("", algo, d, field, iso, dtype, rng.choice([4, 4, 8]), rng.random() < 0.5)
    del c["name"]
    return c


# ---- inputs ---------------------------------------------------------------------------------------------------
def _blobs(dims, gen, count=8):
    """Sum of isotropic Gaussians: centres uniform in the box, sigma uniform in [0.05, 0.15] of the mean side."""
    nx, ny, nz = dims
    u = torch.rand((count, 4), generator=gen, device="cuda")
    side = (nx + ny + nz) / 3.0
    out = torch.zeros((nz, ny, nx), device="cuda")
    axis = [torch.arange(n, device="cuda", dtype=torch.float32) for n in dims]
    for b in range(count):
        s = (0.05 + 0.1 * float(u[b, 3])) * side
        e = [torch.exp(-((axis[a] - float(u[b, a]) * dims[a]) ** 2) / (2 * s * s)) for a in range(3)]
        out.addcmul_(e[2][:, None, None] * e[1][None, :, None], e[0][None, None, :])
    return out


def _noise(dims, gen, octaves=4, period=64):
    """Octaves of trilinearly interpolated uniform [-1, 1] lattices, base period 64 points, gain 0.5."""
    out = torch.zeros(tuple(reversed(dims)), device="cuda")
    for o in range(octaves):
        p = period >> o
        lat = torch.rand([(n - 1) // p + 2 for n in reversed(dims)], generator=gen, device="cuda") * 2 - 1
        for a, n in ((2, dims[0]), (1, dims[1]), (0, dims[2])):
            at = torch.arange(n, device="cuda")
            w = ((at % p).float() / p).reshape([-1 if q == a else 1 for q in range(3)])
            lat = torch.lerp(lat.index_select(a, at // p), lat.index_select(a, at // p + 1), w)
        out.add_(lat, alpha=0.5 ** o)
        del lat
    return out


def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * salt + int(seed))
    return g


def _field(case, seed):
    """(volume [k][j][i], isovalue) of a case; integer samples hold the field over their range."""
    dims = (case["nx"], case["ny"], case["nz"])
    v = _blobs(dims, _gen(seed)) if case["field"] == "blobs" else _noise(dims, _gen(seed))
    iso = case["iso"]
    scale = {"int16": 8192.0, "int8": 60.0, "uint16": 8192.0, "uint8": 60.0}.get(case.get("dtype", "float32"))
    if scale:
        dt = getattr(torch, case["dtype"])
        base = 2.0 if case["dtype"].startswith("u") else 0.0
        top = {"int16": 32767, "int8": 127, "uint16": 65535, "uint8": 255}[case["dtype"]]
        v = v.add_(base).mul_(scale).round_().clamp_(0 if base else -top, top).to(torch.int32).to(dt)
        iso = (iso + base) * scale
    return v, float(np.float32(iso))


_ROOM = {}


def _room(case):
    """Vertices that the caller's buffers hold for a case, the same for every seed: twice the most of three fields
    (three times as many triangles leave room for surfaces cut open at the faces)."""
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _ROOM:
        if case["kind"] == "batch":
            most = max(sum(_cuts(vol, iso) for _, vol, isos in _batch(case, s) for iso in isos) for s in (1, 2))
        else:
            most = max(_cuts(*_field(case, s)) for s in (1, 2, 3))
        _ROOM[key] = 2 * most + 4096
    return _ROOM[key]


def _turned(case, seed):
    """A field whose sign pattern belongs to the case, for results of one size: the seed turns it over along the
    axes and stretches its values by smooth factors in [1, 2]; the isovalue is 0."""
    v, iso = _field(case, case["nx"] + 1000 * case["ny"] + 10 ** 6 * case["nz"])
    v = v.sub_(iso).mul_(_noise((case["nx"], case["ny"], case["nz"]), _gen(seed), 1).mul_(0.5).add_(1.5))
    flips = torch.randint(2, (3,), generator=_gen(seed, 3), device="cuda").tolist()
    return v.flip([a for a in range(3) if flips[a]]).contiguous(), 0.0


def _isos(case):
    return [float(np.float32(-0.4 + 0.8 * (q + 0.5) / case["isos"])) for q in range(case["isos"])]


def _world(case):
    if case.get("unit", True):
        return (1.0, 1.0, 1.0), (0.0, 0.0, 0.0)
    return (0.7, 0.3, 1.1), (-1.0, 2.0, 0.5)


def _batch(case, seed):
    """[(dims, volume, isovalues)]: sides uniform, half blobs and half noise, 1-4 isovalues in [p5, p95]."""
    rng = random.Random(case["sizes"])
    out = []
    for v in range(case["volumes"]):
        dims = tuple(rng.randint(case["least"], case["most"]) for _ in range(3))
        vol = (_blobs if v % 2 == 0 else _noise)(dims, _gen(seed, v + 1))
        some = vol.reshape(-1)[:: max(1, vol.numel() // 65536)].sort().values
        at = [0.05 + 0.9 * rng.random() for _ in range(rng.randint(1, 4))]
        at = torch.tensor([int(a * (some.numel() - 1)) for a in at], device="cuda")
        out.append((dims, vol, [float(x) for x in some[at].tolist()]))
    return out


def _block_stats(vol, dtype):
    """Per 16^3-cell block of a volume (its 17^3 points, clipped at the far faces): min, max and the 32-bin
    histogram over them as fractions of its points, blocks in (z, y, x) order."""
    nz, ny, nx = vol.shape
    cut = [range(0, n - 1, 16) for n in (nz, ny, nx)]
    rows = []
    for z in cut[0]:
        slab = vol[z:z + 17]
        for y in cut[1]:
            band = slab[:, y:y + 17]
            full = [x for x in cut[2] if x + 17 <= nx]
            groups = [band.unfold(2, 17, 16)[:, :, :len(full)].permute(2, 0, 1, 3).reshape(len(full), -1)] if full else []
            groups += [band[:, :, x:x + 17].reshape(1, -1) for x in cut[2] if x + 17 > nx]
            for b in groups:
                lo, hi = b.min(1, keepdim=True).values, b.max(1, keepdim=True).values
                span = hi - lo
                scale = torch.where(span > 0, 32.0 / span, torch.zeros_like(span))
                bins = ((b - lo) * scale).to(torch.int64).clamp_(0, 31)
                h = torch.zeros((b.shape[0], 32), dtype=torch.int64, device=vol.device)
                h.scatter_add_(1, bins, torch.ones_like(bins))
                rows.append(torch.cat([lo.to(dtype), hi.to(dtype), h.to(dtype) / b.shape[1]], 1))
    return torch.cat(rows)


def _train_rows(case, seed):
    """(params, stats, isovalues, targets): blocks of a noise volume, isovalues inside their ranges and
    targets that follow the share of a block's samples near the isovalue."""
    side = 16 * max(2, math.ceil(case["rows"] ** (1 / 3))) + 1
    if side > 273:  # rows beyond the blocks of a 273^3 volume repeat its blocks at other isovalues
        side = 273
    st = _block_stats(_noise((side, side, side), _gen(seed)), torch.float32)
    g = _gen(seed, 7)
    st = st[torch.randint(st.shape[0], (case["rows"],), generator=g, device="cuda")].contiguous()
    u = torch.rand(case["rows"], generator=g, device="cuda")
    iso = st[:, 0] + (st[:, 1] - st[:, 0]) * u.clamp(0.01, 0.99)
    near = torch.gather(st, 1, 2 + (u * 32).long().clamp_(0, 31)[:, None])[:, 0]
    target = near * 40.0 + 0.2 * torch.rand(case["rows"], generator=g, device="cuda")
    fan = [2.0 / 34] * (34 * 64) + [0.0] * 64 + [2.0 / 64] * (64 * 64) + [0.0] * 64 + [1.0 / 64] * 64 + [0.0]
    params = torch.randn(len(fan), generator=g, device="cuda") * torch.tensor(fan, device="cuda").sqrt()
    return params, st, iso.contiguous(), target.contiguous()


# ---- the cases ------------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "mesh":
        vol, iso = _field(case, seed)
        dims = (case["nx"], case["ny"], case["nz"])
        s = {"vol": vol.reshape(-1), "dims": dims, "iso": iso, "algo": ALGOS[case["algo"]]}
        s["spacing"], s["origin"] = _world(case)
        s["out"] = M.DeviceMesh(_room(case), 3 * _room(case), case["index_bytes"])
        for t in (s["out"].points, s["out"].normals, s["out"].tris):
            t.zero_()
        return {"kind": kind, **s}
    if kind == "batch":
        reqs = [M.Request(vol.reshape(-1), dims, iso) for dims, vol, isos in _batch(case, seed) for iso in isos]
        buffers = M.PackedBuffers(_room(case), 3 * _room(case))
        for t in (buffers.points, buffers.normals, buffers.tris):
            t.zero_()
        return {"kind": kind, "requests": reqs, "buffers": buffers}
    if kind == "host":
        vol, iso = _turned(case, seed)
        return {"kind": kind, "image": M.Image3D.from_array(vol.cpu().numpy()), "iso": iso, "algo": ALGOS[case["algo"]]}
    if kind == "size":
        dims = (case["nx"], case["ny"], case["nz"])
        return {"kind": kind, "vol": _noise(dims, _gen(seed)).reshape(-1), "dims": dims, "isos": _isos(case),
                "net": P.Predictor.load()}
    params, st, iso, target = _train_rows(case, seed)
    return {"kind": kind, "params": params, "stats": st, "isos": iso, "target": target,
            "grads": torch.empty(P.N_PARAMS, device="cuda"), "loss": torch.empty(1, device="cuda")}


def run(state):
    kind = state["kind"]
    if kind == "mesh":
        m = M.extract_device(state["vol"], state["dims"], state["iso"], state["algo"], state["spacing"],
                             state["origin"], out=state["out"])
        return m.points, m.normals, m.tris, m.n_points, m.n_tris
    if kind == "batch":
        meshes, b = M.extract_batch_packed(state["requests"], state["buffers"])
        return b.points, b.normals, b.tris, np.array([[m.n_points, m.n_tris] for m in meshes])
    if kind == "host":
        m = M.extract(state["image"], state["iso"], state["algo"])
        return m.points, m.normals, m.triangles.view(np.int64)
    if kind == "size":
        st = P.block_stats(state["vol"], state["dims"])
        return st, state["net"].predict([(st, iso) for iso in state["isos"]])
    return P.mlp_gradient(state["params"], state["stats"], state["isos"], state["target"], state["grads"],
                          state["loss"])


def work(case):
    kind = case["kind"]
    if kind == "train":  # forward, and twice that backward, over 34 -> 64 -> 64 -> 1
        macs = 34 * 64 + 64 * 64 + 64
        return {"bytes": case["rows"] * 4 * 36, "flops": 6 * macs * case["rows"]}
    if kind == "size":
        n = case["nx"] * case["ny"] * case["nz"]
        blocks = math.prod((n1 - 1 + 15) // 16 for n1 in (case["nx"], case["ny"], case["nz"]))
        return {"bytes": 4 * n + blocks * 34 * 4 * (1 + case["isos"]), "flops": 2 * n}
    if kind == "batch":
        total = 0
        for dims, vol, isos in _batch(case, 1):
            for iso in isos:
                v = _cuts(vol, iso)
                total += 4 * vol.numel() + 24 * v + 12 * 2 * v
        return {"bytes": total, "flops": 0}
    vol, iso = _turned(case, 1) if kind == "host" else _field(case, 1)
    v = _cuts(vol, iso)  # vertices; a closed surface has twice as many triangles
    ib = case.get("index_bytes", 8)
    return {"bytes": vol.numel() * vol.element_size() + 24 * v + 3 * ib * 2 * v, "flops": 0}


# ---- the same results in 64 bits, from the definitions ----------------------------------------------------------
def _at_least(vol, iso):
    return (vol if vol.dtype == torch.float32 else vol.to(torch.float32)) >= iso


def _cuts(vol, iso):
    b = _at_least(vol, iso)
    return sum(int((b.narrow(a, 0, b.shape[a] - 1) != b.narrow(a, 1, b.shape[a] - 1)).sum()) for a in range(3))


def _cut_edges(vol, iso):
    """(k, j, axis, i) of every cut edge in Flying Edges order: grid rows in (k, j) order, in a row the x, the y
    and the z edges by i."""
    b = _at_least(vol, iso)
    nz, ny, nx = b.shape
    parts, step = [], max(1, (1 << 28) // (ny * nx))
    for k in range(0, nz, step):
        e = min(nz, k + step)
        m = torch.zeros((e - k, ny, 3, nx), dtype=torch.bool, device=b.device)
        m[:, :, 0, :-1] = b[k:e, :, :-1] != b[k:e, :, 1:]
        m[:, :-1, 1] = b[k:e, :-1] != b[k:e, 1:]
        z = min(e, nz - 1)
        m[:z - k, :, 2] = b[k:z] != b[k + 1:z + 1]
        at = m.nonzero()
        at[:, 0] += k
        parts.append(at)
    return torch.cat(parts)


def _gradient(vol, k, j, i, spacing):
    """Negated central differences, one-sided at the faces, at grid points (x, y, z components)."""
    at, n = [k, j, i], vol.shape
    out = []
    for a, sp in ((2, spacing[0]), (1, spacing[1]), (0, spacing[2])):
        lo, hi = list(at), list(at)
        lo[a], hi[a] = (at[a] - 1).clamp(min=0), (at[a] + 1).clamp(max=n[a] - 1)
        d = vol[tuple(lo)].double() - vol[tuple(hi)].double()
        out.append(d / ((hi[a] - lo[a]).double() * sp))
    return torch.stack(out, 1)


def _vertices(vol, iso, edges, spacing, origin):
    sp, zp = [[float(np.float32(x)) for x in v] for v in (spacing, origin)]
    pts, nrm = [], []
    for e in edges.split(1 << 22):
        k, j, axis, i = e.unbind(1)
        k1, j1, i1 = k + (axis == 2), j + (axis == 1), i + (axis == 0)
        v0, v1 = vol[k, j, i].double(), vol[k1, j1, i1].double()
        w = ((iso - v0) / (v1 - v0))[:, None]
        p = torch.stack([i, j, k], 1).double() + w * torch.nn.functional.one_hot(axis, 3).double()
        pts.append(p * torch.tensor(sp, device=p.device, dtype=p.dtype) + torch.tensor(zp, device=p.device, dtype=p.dtype))
        g0, g1 = _gradient(vol, k, j, i, sp), _gradient(vol, k1, j1, i1, sp)
        nrm.append(g0 + w * (g1 - g0))
    if not pts:
        z = torch.zeros((0, 3), dtype=torch.float64, device=vol.device)
        return z, z
    return torch.cat(pts), torch.cat(nrm)


# Cube edges of each of the 256 cube cases in the order in which its triangles first name them (hexadecimal digits;
# corner v of a cell is bit v of its case): Marching Cubes numbers vertices by cell, then in this order.
_ORDER = (
    "- 038 091 1389 1b2 0381b2 9b20 238b9 32a 02a8 1092a3 12a98 31ba 01b8a 309ab 9b8a 487 4037 091874 49173 "
    "1b2874 37401b2 9b20874 29b734 87432a a7420 9108742a3 4a7921 31ba748 1ba407 4879a0b3 4a79b 945 945038 0451 "
    "84531 1b2945 3801b2459 5b240 25b348 9452a3 02a8459 04512a3 2518a4 ba31945 459018ba 504ab3 584ba 9875 90357 "
    "08715 1357 9875b21 b2190537 82057b 25b37 759832a 97520a 2a308175 a1275 9857b31a 5079a1b a0b3587 a5b7 b56 "
    "03856b 91056b 138956b 1562 1562380 95602 589263 2a3b56 a802b56 0912a356b 56b129a8 6a351 0a8516 36a059 695a8 "
    "56b487 40376b5 10956b874 b5617934 6215487 15263407 87495062 7934256 32a748b56 56b4270a 0914872a356b "
    "912a4756b 87435a16 5a16074 09563a874 695a47 b946 46b9038 b1064 81364b 19426 38019246 0426 82346 b946a32 "
    "028a4b96 32a0614b 614b82a 94631a 81a0694 36a04 684a 76b89 037b96 b76180 b7613 162897 2961703 70862 7236 "
    "2a3b8697 270a96b 1087b62a3 a127b6 86971a3 019a76 70863a 76a 7a6 380a67 091a67 8913a67 b2167a 1b238067a "
    "209b67a 67a23b89 7326 78062 2673091 126897 b6713 b67180 073b96 7b689 648a 3a604 8a64910 96431a 648a21b "
    "1b23a064 48a6092b b3924a6 83246 0246 10924368 14926 83164b b0164 4368b09 b496 4597a6 038459a67 51047a6 "
    "a6784351 945b217a6 67a1b2038459 7a65b420 38452ba67 7326594 94506827 32671054 6827145 945b6173 1b6708945 "
    "4b05367 7b6854 659a8 3a6059 08a516 63a51 1b29a586 03a6951b2 a5860b2 63a52b 598263 96502 1850632 1652 163b859 "
    "b01695 0835b6 b65 ab57 ab57803 57ab109 b57a9183 a2175 0381725a 95720a 725a938 2b537 80257b 91053b72 92817b5 "
    "1537 07815 93057 9785 548ba 540ab3 0918b4a5 b4a5391 2158a4 0a43521 0529a48 95423a 2b5348 52b40 32b584091 "
    "52b419 85431 0541 854390 954 47a9b 038479ab 1ab407 3418b7a 47a921 947a12038 a4720 a47283 2b9734 97b4280 "
    "3b72410 12b847 41973 419708 4307 478 98ba 390ab 0b18a 3b1a 1a298 390a12 0a28 3a2 283b9 92b0 283b01 12b 1839 "
    "019 083 - "
)
# low point offset (x, y, z) and axis of the 12 cube edges
_EDGE = [(0, 0, 0, 0), (1, 0, 0, 1), (0, 1, 0, 0), (0, 0, 0, 1), (0, 0, 1, 0), (1, 0, 1, 1), (0, 1, 1, 0), (0, 0, 1, 1),
         (0, 0, 0, 2), (1, 0, 0, 2), (0, 1, 0, 2), (1, 1, 0, 2)]


def _owned(i0, j0, k0):
    """Edges that a cell numbers first: those no cell before it (smaller k, j, i) has."""
    return [e for e, (dx, dy, dz, a) in enumerate(_EDGE)
            if (dx or a == 0 or i0) and (dy or a == 1 or j0) and (dz or a == 2 or k0)]


def _cell_edges(vol, iso):
    """The cut edges in Marching Cubes order, as _cut_edges gives them in Flying Edges order."""
    b = _at_least(vol, iso)
    table = torch.full((8, 256, 12), -1, dtype=torch.int64)
    for c, order in enumerate(_ORDER.split()):
        for f in range(8):
            own = _owned(f & 1, f & 2, f & 4)
            seq = [int(x, 16) for x in order if x != "-" and int(x, 16) in own]
            table[f, c, :len(seq)] = torch.tensor(seq, dtype=torch.int64)
    table, geo = table.to(b.device), torch.tensor(_EDGE, device=b.device)
    nz, ny, nx = b.shape
    parts, step = [], max(1, (1 << 26) // (ny * nx))
    for k in range(0, nz - 1, step):
        e = min(nz - 1, k + step)
        case = torch.zeros((e - k, ny - 1, nx - 1), dtype=torch.uint8, device=b.device)
        for v, (x, y, z) in enumerate([(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]):
            case |= b[k + z:e + z, y:ny - 1 + y, x:nx - 1 + x].to(torch.uint8) << v
        at = ((case != 0) & (case != 255)).nonzero()
        c = case[at[:, 0], at[:, 1], at[:, 2]].long()
        at[:, 0] += k
        flags = (at[:, 2] == 0).long() + 2 * (at[:, 1] == 0) + 4 * (at[:, 0] == 0)
        edge = table[flags, c]
        cell, slot = (edge >= 0).nonzero().unbind(1)
        g, at = geo[edge[cell, slot]], at[cell]
        parts.append(torch.stack([at[:, 0] + g[:, 2], at[:, 1] + g[:, 1], g[:, 3], at[:, 2] + g[:, 0]], 1))
    return torch.cat(parts)


def _edges(vol, iso, algo):
    if algo == "mc":
        return _cell_edges(vol, iso)
    e = _cut_edges(vol, iso)
    return e if algo == "fe" else e[e[:, 2].sort(stable=True).indices]  # duplicate-free: all x, all y, all z edges


def _net(params, st, iso):
    """The network's output, from its parameters W1 [34][64], b1, W2 [64][64], b2, W3 [64], b3."""
    w1, b1, w2, b2, w3, b3 = params.split([34 * 64, 64, 64 * 64, 64, 64, 1])
    span = st[:, 1] - st[:, 0]
    x = torch.cat([torch.where(span[:, None] > 0, (st[:, :2] - iso[:, None]) / span[:, None], st[:, :2] * 0), st[:, 2:]], 1)
    h = torch.relu(x @ w1.view(34, 64) + b1)
    return torch.relu(h @ w2.view(64, 64) + b2) @ w3 + b3


def _padded(t, rows):
    """The rows of a buffer that a result leaves free stay as they were: zero."""
    return torch.nn.functional.pad(t, (0, 0, 0, rows - t.shape[0]))


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        params, st, iso, target = [t.double() for t in _train_rows(case, seed)]
        params.requires_grad_(True)
        loss = ((_net(params, st, iso) - target) ** 2).mean()
        loss.backward()
        return params.grad, loss.detach().reshape(1)
    if kind == "size":
        # the bins are taken in float32, as the statistics define them, the shares in 64 bits
        st = _block_stats(_noise((case["nx"], case["ny"], case["nz"]), _gen(seed)), torch.float64)
        params = torch.from_numpy(np.fromfile(P.WEIGHTS, np.float32)[3:]).cuda().double()  # margins, then parameters
        got = []
        for iso in _isos(case):
            on = (st[:, 0] < iso) & (st[:, 1] >= iso)
            y = _net(params, st[on], torch.full((int(on.sum()),), iso, dtype=torch.float64, device=st.device))
            got.append(float(torch.relu(y).sum()) * 256.0)  # the network counts in 256s
        return st, got
    if kind == "batch":
        pts, nrm = [], []
        for dims, vol, isos in _batch(case, seed):
            for iso in isos:
                p, n = _vertices(vol, iso, _cut_edges(vol, iso), (1, 1, 1), (0, 0, 0))
                pts.append(p)
                nrm.append(n)
        n = _room(case) + _room(case) // 4  # the package's buffers keep a quarter more
        return _padded(torch.cat(pts), n), _padded(torch.cat(nrm), n), None, None
    vol, iso = _turned(case, seed) if kind == "host" else _field(case, seed)
    if vol.dtype != torch.float32:
        vol = vol.to(torch.float32)
    spacing, origin = _world(case)
    p, n = _vertices(vol, iso, _edges(vol, iso, case["algo"]), spacing, origin)
    if kind == "host":
        return p, n, None
    return _padded(p, _room(case)), _padded(n, _room(case)), None, None, None
