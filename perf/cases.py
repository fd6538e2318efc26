"""The work whose speed is kept track of: one pass each through this framework's public
entry points, on inputs made on the GPU from a seed.

The diffusion itself (``device.diffuse``, ``device.BatchPlan`` and the drop-in
``diffusion`` call) comes at the shapes, kernels and storage types it is used with; the
steps either side of it in the pipeline (sphere morphology before it, field combination
and histograms after it) come at the sizes and bins of the pipeline's blocks.
"""
import numpy as np
import torch

from maxibone_b200 import device, morphology
from maxibone_b200.diffusion import diffusion
from maxibone_b200.fields import combine_fields
from maxibone_b200.histograms import axis_histograms, field_histogram
from maxibone_b200.kernels import gauss_kernel
from maxibone_b200.synthetic import batch_shapes, bone_implant_mask, spheres_mask_torch


def _diffuse(name, shape, sigma, reps, field, packed=False, field_out=True):
    nz, ny, nx = shape
    return {"name": name, "kind": "diffuse", "nz": nz, "ny": ny, "nx": nx, "sigma": sigma, "reps": reps,
            "field": field, "packed": packed, "field_out": field_out}


def listed():
    return [
        # A region of interest at the reference test's size: every launch is short.
        _diffuse("f32_small_128", (128, 128, 128), 3.0, 10, "f32"),
        # A cropped sample whose extents suit no tile and no vector width.
        _diffuse("f32_ragged", (301, 517, 333), 2.5, 10, "f32"),
        # A whole scan in the default (FP32) form, as the reference's in-memory call holds it.
        _diffuse("f32_scan_1024", (1024, 1024, 1024), 8.0, 10, "f32", field_out=False),
        # The same scan with the mask bit-packed and a BF16 field.
        _diffuse("bf16_scan_1024", (1024, 1024, 1024), 8.0, 10, "bf16", packed=True, field_out=False),
        # A crop with an FP16 field; extents are no multiples of the 128-wide tiles.
        _diffuse("f16_crop", (200, 344, 456), 4.0, 20, "f16"),
        # The widest kernel in use, sigma 32 (257 taps).
        _diffuse("bf16_wide_257taps", (256, 512, 768), 32.0, 4, "bf16"),
        # Many samples of uneven size with their own sigma, as one plan.
        {"name": "batch_16", "kind": "batch", "volumes": 16, "shapes_seed": 3, "reps": 10, "field": "bf16"},
        # A pipeline script's call: numpy arrays in pageable memory in and out.
        {"name": "dropin_numpy", "kind": "dropin", "nz": 360, "ny": 400, "nx": 416, "sigma": 3.0, "reps": 10},
        # Mask preparation: the radius that the pipeline's dilate / close / open steps apply over and over.
        {"name": "dilate_u8_r16", "kind": "morphology", "nz": 512, "ny": 1024, "nx": 1024, "radius": 16,
         "dilate": True, "packed": False},
        # The field's consumers at the pipeline's bins: a tomogram against the field at half its resolution ...
        {"name": "field_histogram", "kind": "field_histogram", "nz": 512, "ny": 1024, "nx": 1024, "scale": 2,
         "field_bins": 2048, "voxel_bins": 4096},
        # ... and the x, y, z and radial histograms of one z-block.
        {"name": "axis_histograms", "kind": "axis_histograms", "nz": 128, "ny": 1024, "nx": 1024,
         "voxel_bins": 4096},
        # The Gaussian + EDT combination of a cropped scan.
        {"name": "combine_fields", "kind": "combine", "nz": 384, "ny": 1000, "nx": 1000},
    ]


def _log(rng, lo, hi):
    """An integer between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def _shape(rng, lo, hi, step=1):
    return tuple(max(step, _log(rng, lo, hi) // step * step) for _ in range(3))


def draw(rng):
    kind = rng.choice(["f32", "f32", "16bit", "16bit", "wide", "batch", "dropin", "morphology", "field_histogram",
                       "axis_histograms", "combine"])
    if kind == "f32":
        case = _diffuse("", _shape(rng, 64, 700), round(rng.uniform(1.0, 10.0), 2), _log(rng, 2, 20), "f32",
                        rng.random() < 0.3, rng.random() < 0.5)
    elif kind == "16bit":
        case = _diffuse("", _shape(rng, 64, 640, 8), round(rng.uniform(1.0, 8.0), 2), _log(rng, 2, 40),
                        rng.choice(["bf16", "f16"]), rng.random() < 0.5, rng.random() < 0.5)
    elif kind == "wide":
        case = _diffuse("", _shape(rng, 96, 640, 8), round(rng.uniform(9.0, 32.0), 2), _log(rng, 2, 6),
                        rng.choice(["bf16", "f16"]), rng.random() < 0.5, rng.random() < 0.5)
    elif kind == "batch":
        case = {"kind": "batch", "volumes": rng.randint(3, 24), "shapes_seed": rng.randrange(1 << 16),
                "reps": _log(rng, 2, 20), "field": rng.choice(["bf16", "f16"])}
    elif kind == "dropin":
        nz, ny, nx = _shape(rng, 48, 480)
        case = {"kind": "dropin", "nz": nz, "ny": ny, "nx": nx, "sigma": round(rng.uniform(1.0, 8.0), 2),
                "reps": _log(rng, 2, 20)}
    elif kind == "morphology":
        packed = rng.random() < 0.4
        nz, ny, nx = _shape(rng, 64, 900)
        case = {"kind": "morphology", "nz": nz, "ny": ny, "nx": max(32, nx // 32 * 32) if packed else nx,
                "radius": rng.randint(1, 20), "dilate": rng.random() < 0.5, "packed": packed}
    elif kind == "field_histogram":
        nz, ny, nx = _shape(rng, 64, 900)
        case = {"kind": kind, "nz": nz, "ny": ny, "nx": nx, "scale": rng.choice([1, 2, 2, 4]),
                "field_bins": rng.choice([256, 1024, 2048]), "voxel_bins": rng.choice([512, 2048, 4096])}
    elif kind == "axis_histograms":
        nz, ny, nx = _shape(rng, 64, 900)
        case = {"kind": kind, "nz": min(nz, 256), "ny": ny, "nx": nx, "voxel_bins": rng.choice([512, 2048, 4096])}
    else:
        nz, ny, nx = _shape(rng, 64, 900)
        case = {"kind": kind, "nz": nz, "ny": ny, "nx": nx}
    case.pop("name", None)
    return case


def _dims(case):
    return case["nz"], case["ny"], case["nx"]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _mask(shape, seed, foreground=0.25):
    """An implant in trabecular bone; the implant's radius goes with the sample."""
    return bone_implant_mask(shape, seed=seed, foreground=foreground,
                             implant_radius=0.117 * min(shape[1:]), device="cuda")


def _smooth_field(shape, g):
    """A smooth uint16 field (as int16 bits) with a plateau at 65535, as the diffusion leaves it."""
    coarse = torch.rand((1, 1, *(max(2, n // 40 + 2) for n in shape)), generator=g, device="cuda")
    f = torch.nn.functional.interpolate(coarse, size=shape, mode="trilinear", align_corners=True)[0, 0]
    return f.mul_(1.4).clamp_(0, 1).mul_(65535.0).to(torch.int32).to(torch.int16)


def _tomogram(shape, seed, g):
    """uint16 grey values (as int16 bits): bone with noise, a bright implant, air beside the sample."""
    mask = _mask(shape, seed)
    zz = torch.arange(shape[0], device="cuda", dtype=torch.float32)[:, None, None]
    v = torch.randn(shape, generator=g, device="cuda").mul_(1500.0).add_(19000.0 + 7000.0 * torch.sin(zz * 0.01))
    v.masked_fill_(mask.bool(), 45000.0)
    v[:, :, : shape[2] // 4] = 0.0
    return v.clamp_(0, 65535).to(torch.int32).to(torch.int16)


def _batch_masks(case, seed):
    return [(shape, sigma, spheres_mask_torch(shape, foreground, seed=seed * 1009 + i))
            for i, (shape, sigma, foreground) in enumerate(batch_shapes(case["volumes"], case["shapes_seed"]))]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "diffuse":
        shape = _dims(case)
        mask = _mask(shape, seed)
        if case["packed"]:
            mask = device.bitpack(mask)
        return {"case": case, "mask": mask, "kernel": gauss_kernel(case["sigma"]).astype(np.float32),
                "output": torch.empty(shape, dtype=torch.uint16, device="cuda"),
                "field_out": torch.empty(shape, dtype=torch.float32, device="cuda") if case["field_out"] else None,
                # The FP32 form's size, so that a 16-bit request on a shape without a 16-bit form can run too.
                "workspace": torch.empty(device.workspace_bytes(shape, "f32"), dtype=torch.uint8, device="cuda")}
    if kind == "batch":
        volumes = _batch_masks(case, seed)
        outs = [torch.empty(shape, dtype=torch.uint16, device="cuda") for shape, _, _ in volumes]
        fields = [torch.empty(shape, dtype=torch.float32, device="cuda") for shape, _, _ in volumes]
        plan = device.BatchPlan([m for _, _, m in volumes], [gauss_kernel(s) for _, s, _ in volumes], case["reps"],
                                outputs=outs, field=case["field"], field_outs=fields)
        return {"case": case, "plan": plan, "outputs": outs, "fields": fields}
    if kind == "dropin":
        mask = _mask(_dims(case), seed).cpu().numpy()
        return {"case": case, "mask": mask, "kernel": gauss_kernel(case["sigma"]),
                "output": np.zeros(mask.shape, np.uint16)}
    if kind == "morphology":
        shape = _dims(case)
        # Thin structures to dilate, thicker ones to erode: neither fills or empties the volume at once.
        mask = _mask(shape, seed, 0.06 if case["dilate"] else 0.4)
        if case["packed"]:
            mask = device.bitpack(mask).view(shape[0], shape[1], shape[2] // 32)
        names = ("erode_3d_sphere", "dilate_3d_sphere")
        fn = getattr(morphology, names[bool(case["dilate"])] + ("_bitpacked" if case["packed"] else ""))
        return {"case": case, "fn": fn, "mask": mask, "result": torch.empty_like(mask)}
    g = _generator(seed)
    if kind == "field_histogram":
        shape = _dims(case)
        voxels = _tomogram(shape, seed, g)
        field = _smooth_field(tuple(-(-n // case["scale"]) for n in shape), g)
        bins = torch.zeros((case["field_bins"], case["voxel_bins"]), dtype=torch.int64, device="cuda")
        return {"case": case, "voxels": voxels, "field": field, "bins": bins}
    if kind == "axis_histograms":
        nz, ny, nx = _dims(case)
        n_r = int(np.sqrt((nx // 2) ** 2 + (ny // 2) ** 2)) + 1
        return {"case": case, "voxels": _tomogram((nz, ny, nx), seed, g),
                "bins": [torch.zeros((n, case["voxel_bins"]), dtype=torch.int64, device="cuda")
                         for n in (nx, ny, nz, n_r)]}
    shape = _dims(case)
    gauss, edt = _smooth_field(shape, g), _smooth_field(shape, g)
    return {"case": case, "gauss": gauss, "edt": edt, "output": torch.empty_like(gauss)}


def _bits(u16):
    return u16.view(torch.int16)  # the same memory, in the type torch can index


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "diffuse":
        device.diffuse(state["mask"], state["kernel"], case["reps"], output=state["output"], field=case["field"],
                       field_out=state["field_out"], shape=_dims(case) if case["packed"] else None,
                       workspace=state["workspace"])
        return {"output": _bits(state["output"]), "field": state["field_out"]}
    if kind == "batch":
        state["plan"].run()
        return {"outputs": [_bits(o) for o in state["outputs"]], "fields": state["fields"]}
    if kind == "dropin":
        diffusion(state["mask"], state["kernel"], state["output"], case["reps"])
        return state["output"]
    if kind == "morphology":
        state["fn"](state["mask"], case["radius"], state["result"])
        return state["result"]
    if kind == "field_histogram":
        field_histogram(state["voxels"], state["field"], (0, 0, 0), state["bins"], (1.0, 32000.0), (1.0, 65535.0))
        return state["bins"]
    if kind == "axis_histograms":
        axis_histograms(state["voxels"], (0, 0, 0), *state["bins"], (case["ny"] // 2, case["nx"] // 2),
                        (1.0, 32000.0))
        return state["bins"]
    return combine_fields(state["gauss"], state["edt"], state["output"])


def work(case):
    kind = case["kind"]
    if kind == "batch":
        total = {"bytes": 0, "flops": 0}
        for shape, sigma, _ in batch_shapes(case["volumes"], case["shapes_seed"]):
            n = int(np.prod(shape))
            total["bytes"] += n * (1 + 2 + 4)
            total["flops"] += n * case["reps"] * 3 * 2 * len(gauss_kernel(sigma))
        return total
    n = case["nz"] * case["ny"] * case["nx"]
    if kind in ("diffuse", "dropin"):
        mask = 0.125 if case.get("packed") else 1
        return {"bytes": n * (mask + 2 + (4 if case.get("field_out") else 0)),
                "flops": n * case["reps"] * 3 * 2 * len(gauss_kernel(case["sigma"]))}
    if kind == "morphology":
        return {"bytes": 2 * n // (8 if case["packed"] else 1), "flops": 0}
    if kind == "field_histogram":
        return {"bytes": 2 * n + 2 * n // case["scale"] ** 3 + 8 * case["field_bins"] * case["voxel_bins"], "flops": 0}
    if kind == "axis_histograms":
        n_r = int(np.sqrt((case["nx"] // 2) ** 2 + (case["ny"] // 2) ** 2)) + 1
        return {"bytes": 2 * n + 8 * case["voxel_bins"] * (case["nx"] + case["ny"] + case["nz"] + n_r), "flops": 0}
    return {"bytes": 6 * n, "flops": 0}


def _diffuse_f64(mask, sigma, reps):
    """The repetitions as products with banded matrices in FP64 (zero boundary), masks re-illuminated."""
    taps = gauss_kernel(sigma).astype(np.float32).astype(np.float64)
    r = len(taps) // 2
    bands = []
    for n in mask.shape:
        band = torch.zeros((n, n), dtype=torch.float64, device=mask.device)
        for d in range(-min(r, n - 1), min(r, n - 1) + 1):
            band.diagonal(d).fill_(float(taps[r + d]))
        bands.append(band)
    lit = mask > 0
    f = lit.to(torch.float64)
    for _ in range(reps):
        f = (bands[0] @ f.view(f.shape[0], -1)).view(f.shape)
        f = torch.matmul(bands[1], f)
        f = torch.matmul(f, bands[2].T)
        f.masked_fill_(lit, 1.0)
    return f


def exact(case, seed):
    kind = case["kind"]
    if kind == "diffuse" and case["field_out"]:
        return {"output": None, "field": _diffuse_f64(_mask(_dims(case), seed), case["sigma"], case["reps"])}
    if kind == "batch":
        volumes = _batch_masks(case, seed)
        return {"outputs": [None] * len(volumes),
                "fields": [_diffuse_f64(mask, sigma, case["reps"]) for _, sigma, mask in volumes]}
    return None  # whole numbers only
