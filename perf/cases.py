"""The work users of the encoding have it do, as measurable cases.

Every case goes through the package's public entry points (``PermutoEncoding``, its fused
``forward_mlp`` / ``forward_linear``, ``LatticeAdamW``).  ``what`` names the call:

  infer    features without gradients
  train    forward + backward into the lattice values
  pose     forward + backward into the lattice values and the positions
  normals  forward + gradient to the positions only
  eikonal  forward, position gradient with ``create_graph``, and a backward through both the
           features and that gradient (lattice values and upstream gradient receive theirs)
  adamw    forward + backward + one AdamW step on the lattice values
  linear   inference through the consumer's first layer, Linear(W, 32)
  mlp      inference through a whole small network, W-32-32-32-1 with GELU

``points`` is "uniform" (independent points in a box, what the reference's performance script and
an SDF's free-space samples are) or "rays" (128 consecutive samples along each camera ray).
"""
import math

import numpy as np
import torch

from permutohedral_encoding_b200 import Coarse2Fine, PermutoEncoding
from permutohedral_encoding_b200.optim import LatticeAdamW

DEV = "cuda"
SAMPLES_PER_RAY = 128


def _case(name, what, n, d=3, levels=24, feat=2, capacity=2 ** 18, sigma=1e-4, points="uniform", half=False,
          window=1.0, concat=False):
    c = dict(what=what, n=n, d=d, levels=levels, feat=feat, capacity=capacity, sigma=sigma, points=points, half=half,
             window=window, concat=concat)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the README's usage example: one small query batch, where the latency of a call is what counts
        _case("readme_infer_1000", "infer", 1000),
        # a training step on a small, ragged batch: host work, launches and the dense gradient
        _case("small_train_4099", "train", 4099),
        # dense evaluation of a trained field (the inference half of the performance script)
        _case("infer_1m", "infer", 2 ** 20),
        # the training step of the baseline's main configuration
        _case("train_1m", "train", 2 ** 20),
        # the performance script's variant that also needs position gradients (poses, warp fields)
        _case("pose_512k", "pose", 2 ** 19),
        # the performance script's training loop: step on the table included
        _case("adamw_512k", "adamw", 2 ** 19),
        # SDF training with an eikonal term
        _case("eikonal_512k", "eikonal", 2 ** 19, capacity=2 ** 19),
        # higher-dimensional inputs (time- or view-dependent fields) with a larger table
        _case("dim4_train_1m", "train", 2 ** 20, d=4, levels=16, capacity=2 ** 20, sigma=1e-3),
        _case("dim6_train_1m", "train", 2 ** 20, d=6, levels=16, capacity=2 ** 20, sigma=1e-3),
        # rendering: samples along rays through the fused network, a number of points as it comes
        _case("mlp_rays_1000003", "mlp", 1000003, points="rays"),
        # every option at once: wide fp16 entries, ray samples, a half-open coarse-to-fine window,
        # concatenated points, ragged point and level counts (rows that are no multiple of 32 bytes)
        _case("options_train_300007", "train", 300007, levels=11, feat=4, points="rays", half=True, window=0.6,
              concat=True),
        # the largest step: 2^24 points against a 100 MB table
        _case("train_16m", "train", 2 ** 24, capacity=2 ** 19),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["infer", "train", "train", "pose", "normals", "eikonal", "adamw", "linear", "mlp"])
    d = rng.choice([2, 3, 3, 3, 4, 5, 6, 7])
    feat = rng.choice([2, 2, 2, 4, 8])
    levels = rng.randint(max(4, 16 // feat), 48 // feat)
    n = _log_int(rng, 300, 2 ** 22 if d <= 3 else 2 ** 20)
    if rng.random() < 0.3:
        n = max(256, n // 256 * 256)
    capacity = 2 ** rng.randint(14, 21 - int(math.log2(feat)))
    if rng.random() < 0.15:
        capacity -= rng.randint(1, 1000)
    return _case(None, what, n, d=d, levels=levels, feat=feat, capacity=capacity, sigma=rng.choice([1e-2, 1e-3, 1e-4]),
                 points=rng.choice(["uniform", "rays"]) if d == 3 else "uniform", half=rng.random() < 0.2,
                 window=rng.choice([1.0, 1.0, 1.0, round(rng.uniform(0.3, 0.9), 3)]), concat=rng.random() < 0.2)


def _positions(case, gen):
    n, d = case["n"], case["d"]
    if case["points"] == "uniform":
        half = 1.0 if case["what"] == "eikonal" else 0.5
        return (torch.rand((n, d), device=DEV, generator=gen) * 2 - 1) * half
    # jittered samples at increasing depth along rays from cameras around the scene
    rays = -(-n // SAMPLES_PER_RAY)
    origin = torch.nn.functional.normalize(torch.randn((rays, 1, 3), device=DEV, generator=gen), dim=-1)
    target = (torch.rand((rays, 1, 3), device=DEV, generator=gen) - 0.5) * 0.6
    step = torch.arange(SAMPLES_PER_RAY, device=DEV).view(1, -1, 1)
    t = 0.5 + (step + torch.rand((rays, SAMPLES_PER_RAY, 1), device=DEV, generator=gen)) / SAMPLES_PER_RAY
    return (origin + (target - origin) * t).reshape(-1, 3)[:n].contiguous()


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    torch.manual_seed(seed)
    n, what = case["n"], case["what"]
    enc = PermutoEncoding(case["d"], case["capacity"], case["levels"], case["feat"],
                          np.geomspace(1.0, case["sigma"], case["levels"]), concat_points=case["concat"],
                          half_precision_table=case["half"])
    with torch.no_grad():  # the magnitude of a table that has been trained for a while
        enc.lattice_values.normal_(0.0, 0.1, generator=gen)
    width = enc.output_dims()
    state = dict(what=what, enc=enc, pos=_positions(case, gen), window=None)
    if case["window"] < 1.0:
        state["window"] = Coarse2Fine(case["levels"])(case["window"]).to(device=DEV, dtype=torch.float32)
    if what in ("linear", "mlp"):
        sizes = [width, 32] if what == "linear" else [width, 32, 32, 32, 1]
        mods = []
        for a, b in zip(sizes[:-1], sizes[1:]):
            mods += [torch.nn.Linear(a, b, device=DEV), torch.nn.GELU()]
        state["net"] = mods[0] if what == "linear" else torch.nn.Sequential(*mods[:-1])
    elif what != "infer":
        state["grad"] = torch.randn((n, width), device=DEV, generator=gen)
    if what in ("pose", "normals", "eikonal"):
        state["pos"].requires_grad_(True)
    if what == "eikonal":
        state["up"] = torch.randn((n, width), device=DEV, generator=gen).requires_grad_(True)
        state["dpos"] = torch.randn((n, case["d"]), device=DEV, generator=gen) / n
    if what == "adamw":
        state["opt"] = LatticeAdamW([enc.lattice_values], lr=1e-3, betas=(0.9, 0.99), eps=1e-15, weight_decay=0.0)
        run(state)  # the loop is under way: the moments exist
    return state


def run(state):
    what, enc, pos, window = state["what"], state["enc"], state["pos"], state["window"]
    if what in ("infer", "linear", "mlp"):
        with torch.no_grad():
            if what == "infer":
                return enc(pos, window)
            if what == "linear":
                return enc.forward_linear(pos, state["net"], window)
            return enc.forward_mlp(pos, state["net"], window)

    values = enc.lattice_values
    values.grad = None
    pos.grad = None
    out = enc(pos, window)
    if what == "train":
        out.backward(state["grad"])
        return out.detach(), values.grad
    if what == "pose":
        out.backward(state["grad"])
        return out.detach(), values.grad, pos.grad
    if what == "normals":
        (normal,) = torch.autograd.grad(out, pos, state["grad"])
        return out.detach(), normal
    if what == "eikonal":
        up = state["up"]
        up.grad = None
        (normal,) = torch.autograd.grad(out, pos, up, create_graph=True)
        torch.autograd.backward([out, normal], [state["grad"], state["dpos"]], inputs=[values, up])
        return out.detach(), normal.detach(), values.grad, up.grad
    out.backward(state["grad"])
    state["opt"].step()
    moments = state["opt"].state[values]
    return out.detach(), values.detach(), moments["exp_avg"], moments["exp_avg_sq"]


def work(case):
    n, d, what = case["n"], case["d"], case["what"]
    extra = -(-d // case["feat"]) if case["concat"] else 0
    width = case["feat"] * (case["levels"] + extra)
    entries = min(case["capacity"], n * (d + 1)) * case["levels"] * case["feat"]   # of the table, touched at most
    dense = case["capacity"] * case["levels"] * case["feat"]
    read_table = entries * (2 if case["half"] else 4)
    rows, pos = 4 * n * width, 4 * n * d
    out = {"linear": 4 * n * 32, "mlp": 4 * n}.get(what, rows)
    total = pos + read_table + out
    if what != "infer" and what not in ("linear", "mlp"):
        total += rows                        # upstream gradient
    if what in ("train", "pose", "eikonal", "adamw"):
        total += 4 * dense                   # gradient of the table (the step of adamw reads what it wrote)
    if what in ("pose", "normals", "eikonal"):
        total += pos
    if what == "eikonal":
        total += 2 * rows + pos              # second upstream gradient and its own gradient, d loss / d normal
    if what == "adamw":
        total += 4 * dense * 5               # both moments in and out, values out
    # locating the simplex (elevate, round, rank, weights) and one multiply-add per vertex and feature
    locate, blend = 12 * (d + 1) + d * (d + 1), 2 * (d + 1) * case["feat"]
    passes = {"train": 2, "pose": 3, "normals": 2, "eikonal": 6, "adamw": 2}.get(what, 1)
    flops = n * case["levels"] * (locate + passes * blend)
    if what in ("linear", "mlp"):
        flops += 2 * n * (width * 32 + (2 * 32 * 32 + 32 if what == "mlp" else 0))
    if what == "adamw":
        flops += 12 * dense
    return {"bytes": total, "flops": flops}


def tolerance(case):
    if case["what"] in ("linear", "mlp"):
        return {"rel": 2e-3}                 # operands rounded to tf32 (2^-11), layer after layer
    if case["what"] == "adamw":
        # the step divides the first moment by the root of the second: an entry whose gradient is a
        # cancelling sum may move by up to lr = 1e-3 in the other direction (values are 0.1 rms)
        return {"rel": 1e-4, "max": 0.1}
    return {"rel": 1e-5}                     # 32-bit sums
