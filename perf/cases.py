"""Performance cases: the calls a segmentation program makes of this framework, over the sizes
and types it makes them for.

Every case runs through the Python entry points of `nsgb` (imreconstruct, chain, chain_batch,
BatchPlan, imfillHoles, bwselect, bwlabel2, bwareaopen2, bounding_boxes, morphOpen,
nucleus_candidates, distanceTransform, imhmin and the autograd binding of the float
reconstruction).  Inputs are made on the GPU from the seed: tiles with a bright noisy background
(185 .. 215) and dark elliptical nuclei (40 .. 90, semi-axes 4 .. 20 px, one per 2800 px), the
shapes and values of the repository's synthetic tiles.

`listed()` is the fixed set, `draw(rng)` gives another case of the same ranges, `prepare` makes
the inputs and the plan a program keeps, `run` is one pass, `work` the bytes it cannot do
without, `exact` the outputs of the floating cases from plain torch in 64 bits.
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "emory-cci-fast-ia-gsoc_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import nsgb  # noqa: E402
from nsgb.autograd import imreconstruct_f32  # noqa: E402

DEV = "cuda"
FLT_MAX = torch.finfo(torch.float32).max
TORCH = {"u8": torch.uint8, "u16": torch.uint16, "i32": torch.int32, "f32": torch.float32}
SIZE = {"u8": 1, "u16": 2, "i32": 4, "f32": 4}
SCALE = {"u8": 1, "u16": 257, "i32": 1000, "f32": 1}  # grey levels per u8 level
DROP = 10  # the marker is the mask lowered by this many u8 levels


def listed():
    return [
        # one small field of view: a preview or a cropped region, where launches and latency count
        {"name": "recon_u8_256", "kind": "recon", "dtype": "u8", "rows": 256, "cols": 256, "conn": 8, "erode": False},
        # a 16-bit scanner tile of odd size, 4-connected
        {"name": "recon_u16_1531x2049", "kind": "recon", "dtype": "u16", "rows": 1531, "cols": 2049, "conn": 4,
         "erode": False},
        # clean-up of a nucleus mask of ragged size: binary hole fill, selection and binary reconstruction
        {"name": "masks_u8_1023x1531", "kind": "masks", "rows": 1023, "cols": 1531},
        # the segmentation chain on one full tile (the benchmark's own call)
        {"name": "chain_u8_4096", "kind": "chain", "dtype": "u8", "rows": 4096, "cols": 4096},
        # a slide's uneven tiles as one call, nothing kept between calls
        {"name": "batch_u8_15", "kind": "batch", "dtype": "u8", "tiles": 15, "keep": False},
        # the same with the plan kept and its marker buffers refilled, 32-bit pixels
        {"name": "batch_i32_20", "kind": "batch", "dtype": "i32", "tiles": 20, "keep": True},
        # nucleus candidates of a tile: opening by the 19 x 19 disk, then the candidate stage
        {"name": "s1_u8_4096", "kind": "s1", "rows": 4096, "cols": 4096},
        # watershed input of a tile: distance basins of the nucleus mask and their h-minima
        {"name": "basins_u8_4096", "kind": "basins", "rows": 4096, "cols": 4096, "basins": True},
        # objects of a tile: raster labels, area filter, bounding boxes
        {"name": "objects_u8_4096", "kind": "objects", "rows": 4096, "cols": 4096},
        # a whole low-magnification slide: grey hole fill, threshold, labels
        {"name": "fill_label_u8_16384", "kind": "fill_label", "dtype": "u8", "rows": 16384, "cols": 16384, "conn": 4},
        # grey hole fill of one 32-bit image of odd size, 8-connected
        {"name": "fill_i32_5003x4099", "kind": "fill", "dtype": "i32", "rows": 5003, "cols": 4099, "conn": 8},
        # a training step through the float reconstruction: forward and both gradients
        {"name": "grad_f32_16x2048", "kind": "grad", "batch": 16, "rows": 2048, "cols": 2048, "conn": 8},
    ]


def _side(rng, lo, hi):
    """A side spread over the logarithm of its range; half of them odd, the rest of any remainder."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, v | 1) if rng.random() < 0.5 else v


def draw(rng):
    kind = rng.choice(["recon", "masks", "chain", "batch", "s1", "basins", "objects", "fill_label", "fill", "grad"])
    if kind == "batch":
        return {"kind": kind, "dtype": rng.choice(["u8", "u16", "i32"]), "tiles": rng.randint(3, 20 if rng.random() < 0.5 else 15),
                "keep": rng.random() < 0.5, "salt": rng.randrange(1000)}
    if kind == "grad":
        return {"kind": kind, "batch": rng.choice([1, 2, 4, 8, 16]), "rows": _side(rng, 128, 2048),
                "cols": _side(rng, 128, 2048), "conn": rng.choice([4, 8])}
    hi = {"fill_label": 12000, "fill": 5000}.get(kind, 4096)
    c = {"kind": kind, "rows": _side(rng, 256, hi), "cols": _side(rng, 256, hi)}
    if kind == "recon":
        c.update(dtype=rng.choice(["u8", "u16", "i32", "f32"]), conn=rng.choice([4, 8]), erode=rng.random() < 0.3)
    elif kind == "chain":
        c.update(dtype=rng.choice(["u8", "u16", "i32"]))
    elif kind in ("fill", "fill_label"):
        c.update(dtype=rng.choice(["u8", "u16", "i32"]), conn=rng.choice([4, 8]))
    elif kind == "basins":
        c.update(basins=rng.random() < 0.7)
    return c


# ------------------------------------------------------------------------------------------
# Inputs.

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _tile(rows, cols, g):
    """An int32 tile: background 185 .. 215, dark ellipses of 40 .. 90 (the darker of two that overlap)."""
    img = torch.empty(rows * cols + 1, dtype=torch.int32, device=DEV)  # the last word takes what falls outside
    img.random_(185, 216, generator=g)
    n = max(1, round(rows * cols / 2800))
    u = torch.rand((6, n), generator=g, device=DEV)
    cx, cy = u[0] * cols, u[1] * rows
    a, b = 4 + 16 * u[2], 4 + 16 * u[3]
    c, s = torch.cos(math.pi * u[4]), torch.sin(math.pi * u[4])
    val = (40 + 51 * u[5]).to(torch.int32)
    d = torch.arange(-21, 22, device=DEV)
    for k in range(0, n, 8192):
        q = slice(k, min(n, k + 8192))
        x = (cx[q].long()[:, None] + d)[:, None, :]
        y = (cy[q].long()[:, None] + d)[:, :, None]
        dx, dy = x - cx[q, None, None], y - cy[q, None, None]
        e, f, cc, ss = a[q, None, None], b[q, None, None], c[q, None, None], s[q, None, None]
        inside = ((dx * cc + dy * ss) / e) ** 2 + ((dy * cc - dx * ss) / f) ** 2 <= 1
        inside = inside & (x >= 0) & (x < cols) & (y >= 0) & (y < rows)
        at = torch.where(inside, y * cols + x, rows * cols)
        img.scatter_reduce_(0, at.reshape(-1), val[q, None, None].expand(at.shape).reshape(-1), "amin")
    return img[:-1].view(rows, cols)


def _as(t, dtype):
    return (t * SCALE[dtype]).to(TORCH[dtype])


def _marker(t, dtype, erode=False):
    """The tile lowered (raised for the dual) by DROP levels, within the type's range."""
    return _as((t + DROP).clamp_(max=255) if erode else (t - DROP).clamp_(min=0), dtype)


def _nuclei(t):
    return (t < 128).to(torch.uint8) * 255


def _batch_sizes(case):
    """Heights and widths of 256 .. 4096, the same for every seed (they are the case's own)."""
    import random

    r = random.Random("%s %s %s" % (case["tiles"], case["dtype"], case.get("salt", 0)))
    return [(r.randint(256, 4096), r.randint(256, 4096)) for _ in range(case["tiles"])]


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    st = {"case": dict(case)}
    if kind == "batch":
        sizes = _batch_sizes(case)
        tiles = [_tile(h, w, g) for h, w in sizes]
        st["masks"] = [_as(t, case["dtype"]) for t in tiles]
        # the markers of a batch lie in one buffer, as a reader that fills it in one copy has them
        st["source"] = torch.cat([_marker(t, case["dtype"]).view(-1) for t in tiles])
        own = st["source"].clone() if case["keep"] else st["source"]
        at, views = 0, []
        for h, w in sizes:
            views.append(own[at:at + h * w].view(h, w))
            at += h * w
        st["markers"] = views
        if case["keep"]:
            st["buffer"] = own
            st["plan"] = nsgb.BatchPlan(views, st["masks"])
        return st
    if kind == "grad":
        shape = (case["batch"], case["rows"], case["cols"])
        mask = torch.rand(shape, generator=g, device=DEV)
        st["mask"] = mask.requires_grad_()
        st["marker"] = (mask.detach() * torch.empty(shape, device=DEV).uniform_(0.5, 1.0, generator=g)).requires_grad_()
        st["grad"] = torch.randn(shape, generator=g, device=DEV)
        return st
    rows, cols = case["rows"], case["cols"]
    t = _tile(rows, cols, g)
    if kind == "recon":
        if case["dtype"] == "f32":
            t = t + torch.rand((rows, cols), generator=g, device=DEV)
            st["mask"] = t
            st["marker"] = t + DROP if case["erode"] else t - DROP
        else:
            st["mask"] = _as(t, case["dtype"])
            st["marker"] = _marker(t, case["dtype"], case["erode"])
    elif kind == "chain":
        st["mask"], st["marker"] = _as(t, case["dtype"]), _marker(t, case["dtype"])
    elif kind == "masks":
        st["bin"] = _nuclei(t)
        # single dropped pixels inside the nuclei, and seeds on the darker half of them
        st["bin"][torch.rand((rows, cols), generator=g, device=DEV) < 0.02] = 0
        st["seeds"] = (t < 65).to(torch.uint8) * 255
    elif kind == "s1":
        st["rc"] = (255 - t).to(torch.uint8)
        st["rbc"] = _nuclei(_tile(rows, cols, g))
        st["disk"] = nsgb.disk19()
    elif kind in ("basins", "objects"):
        st["bin"] = _nuclei(t)
    else:
        st["image"] = _as(t, case["dtype"])
    return st


# ------------------------------------------------------------------------------------------
# One pass.

def _out(v):
    """An output to compare: 16-bit planes as int16 words (torch indexes no uint16)."""
    if isinstance(v, dict):
        return {k: _out(x) for k, x in v.items()}
    if isinstance(v, list):
        return [_out(x) for x in v]
    return v.view(torch.int16) if isinstance(v, torch.Tensor) and v.dtype == torch.uint16 else v


def run(st):
    return _out(_pass(st))


def _pass(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "recon":
        return nsgb.imreconstruct(st["marker"], st["mask"], case["conn"], erode=case["erode"])
    if kind == "masks":
        return {"filled": nsgb.imfillHoles(st["bin"], True, 4), "selected": nsgb.bwselect(st["bin"], st["seeds"], 8),
                "grown": nsgb.imreconstructBinary(st["seeds"], st["bin"], 8)}
    if kind == "chain":
        return nsgb.chain(st["marker"], st["mask"], thr=128 * SCALE[case["dtype"]])
    if kind == "batch":
        thr = 128 * SCALE[case["dtype"]]
        if not case["keep"]:
            r = nsgb.chain_batch(st["markers"], st["masks"], thr=thr)
            return {"recon": [x["recon"] for x in r], "fill": [x["fill"] for x in r],
                    "labels": [x["labels"] for x in r], "area": [x["area"] for x in r],
                    "counts": torch.tensor([[x["n_labels"], x["n_kept"]] for x in r])}
        plan = st["plan"]
        st["buffer"].copy_(st["source"])
        nl, nk = plan.chain(thr=thr)
        return {"recon": st["buffer"], "fill": plan.fill, "labels": plan.labels, "area": plan.area,
                "counts": torch.tensor([nl, nk])}
    if kind == "s1":
        opened = nsgb.morphOpen(st["rc"], st["disk"])
        seg, kept = nsgb.nucleus_candidates(st["rc"], opened, st["rbc"])
        return {"opened": opened, "seg": seg, "kept": kept}
    if kind == "basins":
        d = nsgb.distanceTransform(st["bin"], basins=case["basins"])
        return {"distance": d, "minima": nsgb.imhmin(d, 1.0, 8)} if case["basins"] else {"distance": d}
    if kind == "objects":
        labels, n = nsgb.bwlabel2_count(st["bin"], 8)
        kept, n_kept = nsgb.bwareaopen2(st["bin"], False, True, 11, 1000, 8)
        boxes = nsgb.bounding_boxes(labels)
        # the caller's table of a fixed number of rows
        boxes = torch.nn.functional.pad(boxes, (0, case["rows"] * case["cols"] // 64 - boxes.shape[1]))
        return {"labels": labels, "n": n, "kept": kept, "n_kept": n_kept, "boxes": boxes}
    if kind == "fill":
        return nsgb.imfillHoles(st["image"], False, case["conn"])
    if kind == "fill_label":
        filled = nsgb.imfillHoles(st["image"], False, case["conn"])
        bw = nsgb.threshold(filled, 128 * SCALE[case["dtype"]])
        return {"filled": filled, "bw": bw, "labels": nsgb.bwlabel2(bw, 8, True)}
    out = imreconstruct_f32(st["marker"], st["mask"], case["conn"])
    dmarker, dmask = torch.autograd.grad(out, (st["marker"], st["mask"]), st["grad"])
    return {"out": out, "dmarker": dmarker, "dmask": dmask}


def work(case):
    """Bytes of one pass, each input of a call read once and each output written once.  No
    operation count bounds any of these: they compare and move pixels."""
    kind = case["kind"]
    if kind == "batch":
        px = sum(h * w for h, w in _batch_sizes(case))
        return {"bytes": px * (3 * SIZE[case["dtype"]] + 6), "flops": 0}
    px = case["rows"] * case["cols"]
    per = {
        "recon": lambda: 3 * SIZE[case["dtype"]],            # marker, mask; result
        "masks": lambda: 2 + 3 + 3,                           # fill; image, seeds, result twice
        "chain": lambda: 3 * SIZE[case["dtype"]] + 6,         # ... and fill, labels, area
        "s1": lambda: 2 + 4,                                  # opening; rc, opened, rbc, seg
        "basins": lambda: 1 + 4 + (8 if case["basins"] else 0),
        "objects": lambda: 5 + 2 + 4,                         # labels; area filter; boxes
        "fill": lambda: 2 * SIZE[case["dtype"]],
        "fill_label": lambda: 2 * SIZE[case["dtype"]] + SIZE[case["dtype"]] + 1 + 5,
        "grad": lambda: case["batch"] * 24,                   # marker, mask, out; g, dmarker, dmask
    }[kind]()
    return {"bytes": px * per, "flops": 0}


# ------------------------------------------------------------------------------------------
# The floating outputs from plain torch.  A reconstruction only copies input values, so it is
# iterated pixel-wise to its fixed point; distances and gradients are summed in 64 bits.

def _neighbours(conn):
    near = [(-1, 0), (1, 0), (0, -1), (0, 1)]
    return near + ([(-1, -1), (-1, 1), (1, -1), (1, 1)] if conn == 8 else [])


def _shifted(t, dy, dx, fill):
    """t read at (y + dy, x + dx), `fill` outside."""
    h, w = t.shape[-2:]
    out = torch.full_like(t, fill)
    out[..., max(0, -dy):h - max(0, dy), max(0, -dx):w - max(0, dx)] = \
        t[..., max(0, dy):h - max(0, -dy), max(0, dx):w - max(0, -dx)]
    return out


def _dilate(r, conn):
    """Max over a pixel and its neighbours, the ring around the image 0."""
    p = torch.nn.functional.pad(r, (1, 1, 1, 1), value=0.0)
    if conn == 8:
        p = torch.maximum(torch.maximum(p[..., :-2], p[..., 1:-1]), p[..., 2:])
        return torch.maximum(torch.maximum(p[..., :-2, :], p[..., 1:-1, :]), p[..., 2:, :])
    c = torch.maximum(torch.maximum(p[..., :-2, 1:-1], p[..., 1:-1, 1:-1]), p[..., 2:, 1:-1])
    return torch.maximum(torch.maximum(p[..., 1:-1, :-2], p[..., 1:-1, 2:]), c)


def _reconstruct(marker, mask, conn):
    r = torch.minimum(marker, mask)
    while True:
        before = r
        for _ in range(16):
            r = torch.minimum(_dilate(r, conn), mask)
        if torch.equal(r, before):
            return r


def _exact_grad(case, st):
    mask, marker, g = st["mask"].detach(), st["marker"].detach(), st["grad"]
    b, h, w = mask.shape
    n = h * w
    r = _reconstruct(marker, mask, case["conn"])
    q = torch.arange(n, dtype=torch.int32, device=DEV).view(1, h, w)
    border = torch.zeros((1, h, w), dtype=torch.bool, device=DEV)
    border[:, 0], border[:, -1], border[:, :, 0], border[:, :, -1] = True, True, True, True
    key = torch.where(border & (r == 0), 2 * n, torch.full_like(r, 2 * n + 1, dtype=torch.int32))
    key = torch.where(r == marker, n + q, key)
    key = torch.where(r == mask, q.expand_as(key), key).to(torch.int32)
    # the smallest source of each plateau (connected pixels of one result value)
    while True:
        before = key
        for dy, dx in _neighbours(case["conn"]):
            near = _shifted(key, dy, dx, 2 * n + 1)
            key = torch.where(_shifted(r, dy, dx, float("nan")) == r, torch.minimum(key, near), key)
        if torch.equal(key, before):
            break
    # mask sources in 0 .. n-1, marker sources in n .. 2n-1, the ring's constant in the last
    total = torch.zeros((b, 2 * n + 2), dtype=torch.float64, device=DEV)
    total.scatter_add_(1, key.view(b, -1).long(), g.double().view(b, -1))
    return {"out": r.double(), "dmarker": total[:, n:2 * n].reshape(b, h, w), "dmask": total[:, :n].reshape(b, h, w)}


def _exact_basins(case, st):
    m = st["bin"] != 0
    h, w = m.shape
    far = float(h + w)
    y = torch.arange(h, dtype=torch.float64, device=DEV).view(h, 1).expand(h, w)
    up = y - torch.cummax(torch.where(m, torch.full_like(y, -far), y), 0).values
    down = -y - torch.cummax(torch.where(m, torch.full_like(y, -2 * far), -y).flip(0), 0).values.flip(0)
    g2 = torch.minimum(torch.minimum(up, down), torch.full_like(up, far)).square()
    best, k = g2, 1
    while k < w and k * k < float(best.max()):
        for dx in (-k, k):
            best = torch.minimum(best, _shifted(g2, 0, dx, math.inf) + k * k)
        k += 1
    d = best.sqrt()
    if not case["basins"]:
        return {"distance": d}
    basins = torch.where(m, -d, torch.full_like(d, -FLT_MAX))
    inverted = -basins
    return {"distance": basins, "minima": -_reconstruct(inverted - 1.0, inverted, 8)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "grad":
        return _exact_grad(case, prepare(case, seed))
    if kind == "basins":
        return _exact_basins(case, prepare(case, seed))
    if kind == "recon" and case["dtype"] == "f32":
        st = prepare(case, seed)
        if case["erode"]:
            # the dual, with no ring: values well below 0 after the change of sign
            top = -st["mask"].double()
            return -(_reconstruct(-st["marker"].double() + 1024, top + 1024, case["conn"]) - 1024)
        return _reconstruct(st["marker"].double(), st["mask"].double(), case["conn"])
    return None  # whole numbers
