"""Performance cases of the framework: what its users call, over the sizes they call it with.

Every case goes through the public Python front end (`dmtz_gb300.Context`, `dmtz_gb300.Network`).
Fields are the repository's synthetic ones: Gaussian mixtures and power-law random fields, with
uniform or SZ-style decompression error.  Device-resident fields are edited in place by the
correction, so a pass first copies the decompressed field back into the working buffer; the
context runs on its own stream, so the copy is waited for before the call.
"""
import math

import numpy as np
import torch

import dmtz_gb300 as dm
from dmtz_gb300 import synth

FULL_MSC = (1, 1, 1, 0, 0, 0, 0)
EXTREMA = (0, 0, 0, 0, 0, 0, 0)


def listed():
    return [
        # a call on a handful of vertices: launches, synchronisations and host work
        dict(name="correct_tiny", kind="correct_host", field="gauss", err="uniform", W=16, H=16, D=16, eps=1e-2,
             msc=True, graph=0, strict=False),
        # the small plain method: extrema only, 64^3 Gaussian mixture, eps 1e-3
        dict(name="correct_extrema_64", kind="correct_host", field="gauss", err="uniform", W=64, H=64, D=64, eps=1e-3,
             msc=False, graph=0, strict=False),
        # a strongly disturbed field of ragged size: hundreds of rounds with short lists
        dict(name="correct_noisy", kind="correct_dev", field="gauss", err="uniform", W=97, H=61, D=75, eps=1e-2,
             msc=True, graph=1, strict=False),
        # whole-path separatrix checks on a ragged field
        dict(name="correct_strict", kind="correct_dev", field="powerlaw", err="sz", W=120, H=89, D=101, eps=1e-3,
             msc=True, graph=1, strict=True),
        # the headline workload: 256^3 power-law field, SZ-style error, full Morse-Smale complex
        dict(name="correct_msc_256", kind="correct_dev", field="powerlaw", err="sz", W=256, H=256, D=256, eps=1e-4,
             msc=True, graph=1, strict=False),
        # many fields of uneven sizes and both value types in one call
        dict(name="correct_batch", kind="batch", n=8, lo=32, hi=96, sizes=2024, workers=8),
        # gradient pairing of one field, handed back to the host in the reference's layout
        dict(name="extract", kind="extract", field="powerlaw", W=120, H=97, D=83),
        # manifold labels of one field, handed back to the host
        dict(name="labels", kind="labels", field="gauss", W=96, H=121, D=70),
        # acceptance check of a result: separatrix labels and critical cells against the original's
        dict(name="agreement", kind="agreement", field="powerlaw", err="sz", W=160, H=144, D=129, eps=1e-3),
        # the learned proposal's input features
        dict(name="features", kind="features", field="powerlaw", err="sz", W=160, H=144, D=128, eps=1e-4),
        # the learned proposal's network, inference on a ragged grid
        dict(name="net_forward", kind="net_forward", W=161, H=127, D=110),
        # one training pass of the network: forward, loss, gradients of every parameter
        dict(name="net_train", kind="net_train", W=100, H=75, D=53),
    ]


def _dims(rng, lo, hi, most):
    """Three extents, log-uniform in [lo, hi], with at most `most` vertices."""
    while True:
        d = [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(3)]
        if d[0] * d[1] * d[2] <= most:
            return dict(W=d[0], H=d[1], D=d[2])


def draw(rng):
    kind = rng.choice(["correct_host", "correct_dev", "correct_dev", "batch", "extract", "labels", "agreement",
                       "features", "net_forward", "net_train"])
    if kind in ("correct_host", "correct_dev"):
        field, err = rng.choice([("gauss", "uniform"), ("powerlaw", "sz")])
        eps = rng.choice([1e-2, 1e-3, 1e-4])
        most = 440_000 if eps > 5e-3 else 2_000_000
        c = dict(kind=kind, field=field, err=err, eps=eps, msc=rng.random() < 0.8, graph=rng.choice([0, 1]),
                 strict=rng.random() < 0.25, **_dims(rng, 12, 96 if kind == "correct_host" else 256, most))
        return c
    if kind == "batch":
        lo = rng.randint(16, 40)
        return dict(kind=kind, n=rng.randint(2, 8), lo=lo, hi=rng.randint(lo + 8, 96), sizes=rng.randint(0, 1 << 20),
                    workers=rng.choice([2, 4, 8]))
    if kind in ("extract", "labels"):
        return dict(kind=kind, field=rng.choice(["gauss", "powerlaw"]), **_dims(rng, 12, 160, 1_500_000))
    if kind in ("agreement", "features"):
        return dict(kind=kind, field="powerlaw", err="sz", eps=rng.choice([1e-3, 1e-4]),
                    **_dims(rng, 16, 224, 4_000_000))
    return dict(kind=kind, **_dims(rng, 16, 200, 2_500_000 if kind == "net_forward" else 500_000))


# ------------------------------------------------------------------ inputs
def _field(kind, dims, seed):
    """One original field as a flat float64 device tensor."""
    if kind == "powerlaw":
        return synth.power_law_device(dims, seed)
    scale = (dims[0] + dims[1] + dims[2]) / 3.0 / 64.0
    return synth.gaussian_mix_device(dims, seed, n_gauss=32, sigma=(2.0 * scale, 8.0 * scale)).float().double()


def _decompressed(f, err, rel_eps, seed):
    """f with a bounded decompression error, as synth's models make it."""
    gen = torch.Generator(device=f.device)
    gen.manual_seed(seed + 7919)
    eps = rel_eps * float((f.max() - f.min()).item())
    noise = (2.0 * torch.rand(f.shape, generator=gen, device=f.device, dtype=torch.float64) - 1.0) * eps
    if err == "uniform":
        return f + noise
    sel = torch.rand(f.shape, generator=gen, device=f.device, dtype=torch.float64) < 0.05
    fmin = f.min()
    g = fmin + 2.0 * eps * torch.round((f - fmin) / (2.0 * eps)) + sel * noise
    return torch.maximum(torch.minimum(g, f + eps), f - eps)


def _extents(case):
    return case["W"], case["H"], case["D"]


def _batch_dims(case):
    r = np.random.Generator(np.random.PCG64(case["sizes"]))
    return [tuple(int(x) for x in r.integers(case["lo"], case["hi"] + 1, size=3)) for _ in range(case["n"])]


def _net_input(case, seed):
    """Features of the kind the network meets: differences squashed to (-1, 1), a sparse mismatch bit."""
    V = case["W"] * case["H"] * case["D"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 31)
    feat = torch.tanh(torch.randn((V, 16), generator=gen, device="cuda"))
    feat[:, 1] = (torch.rand(V, generator=gen, device="cuda") < 0.05).float()
    target = torch.tanh(torch.randn(V, generator=gen, device="cuda"))
    active = (torch.rand(V, generator=gen, device="cuda") < 0.4).to(torch.uint8)
    active[::97] = 8  # vertices the exact loop changed weigh more
    return feat.to(torch.bfloat16).contiguous(), target.contiguous(), active.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    seed = int(seed)
    s = dict(case=case)
    if kind in ("net_forward", "net_train"):
        s["net"] = dm.Network(seed=seed)
        s["feat"], s["target"], s["active"] = _net_input(case, seed)
        s["out"] = torch.empty(case["W"] * case["H"] * case["D"], dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        return s
    s["ctx"] = dm.Context()
    if kind == "batch":
        s["fields"] = []
        for i, dims in enumerate(_batch_dims(case)):
            field, err = (("gauss", "uniform"), ("powerlaw", "sz"))[(i // 2) % 2]
            rel = (1e-3, 1e-4)[i % 2] if field == "powerlaw" else (1e-2, 1e-3)[i % 2]
            f = _field(field, dims, seed + 13 * i)
            g = _decompressed(f, err, rel, seed + 13 * i)
            dt = np.float32 if i % 2 == 0 else np.float64
            shape = (dims[2], dims[1], dims[0])
            s["fields"].append((f.cpu().numpy().astype(dt).reshape(shape), g.cpu().numpy().astype(dt).reshape(shape),
                                rel))
        return s
    dims = _extents(case)
    f = _field(case["field"], dims, seed)
    if kind in ("extract", "labels"):
        s["f"] = f.cpu().numpy()
        return s
    g = _decompressed(f, case["err"], case["eps"], seed)
    if kind == "correct_host":
        s["f"], s["g"] = f.cpu().numpy(), g.cpu().numpy()
        return s
    s["f"], s["g0"], s["g"] = f, g, g.clone()
    if kind == "features":
        s["feat"] = torch.empty((f.numel(), 16), dtype=torch.bfloat16, device="cuda")
        s["active"] = torch.empty(f.numel(), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ one pass
def _counts(rep):
    """The report's whole numbers that describe the result."""
    return np.array([rep["outer_iterations"], rep["cp_rounds"], rep["path_rounds"], rep["edited_vertices"],
                     rep["stall_breaks"], rep["converged"], *rep["initial_mismatch"]], np.int64)


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "correct_host":
        out, rep, cnt = s["ctx"].correct(s["f"], s["g"], c["eps"], FULL_MSC if c["msc"] else EXTREMA, dims=_extents(c),
                                         use_graph=c["graph"], return_counter=True, strict=c["strict"])
        return {"field": out, "edits": cnt, "counts": _counts(rep)}
    if kind == "correct_dev":
        s["g"].copy_(s["g0"])
        torch.cuda.synchronize()
        rep = s["ctx"].correct_ptr(s["f"].data_ptr(), s["g"].data_ptr(), _extents(c), c["eps"],
                                   FULL_MSC if c["msc"] else EXTREMA, True, use_graph=c["graph"], strict=c["strict"])
        return {"field": s["g"], "counts": _counts(rep)}
    if kind == "batch":
        res = s["ctx"].correct_batch(s["fields"], FULL_MSC, workers=c["workers"])
        return [{"field": out, "counts": _counts(rep), "status": st} for out, rep, st in res]
    if kind == "extract":
        return list(s["ctx"].extract(s["f"], dims=_extents(c)))
    if kind == "labels":
        return list(s["ctx"].labels(s["f"], dims=_extents(c)))
    if kind == "agreement":
        r = s["ctx"].separatrix_agreement(s["f"].data_ptr(), s["g0"].data_ptr(), _extents(c), on_device=True)
        return {k: int(v) for k, v in r.items()}
    if kind == "features":
        s["ctx"].features(s["f"].data_ptr(), s["g0"].data_ptr(), _extents(c), c["eps"], s["feat"].data_ptr(),
                          s["active"].data_ptr())
        return {"error": s["feat"][:, 0], "mismatch": s["feat"][:, 1], "slopes": s["feat"][:, 2:],
                "active": s["active"]}
    net, dims = s["net"], _extents(c)
    if kind == "net_forward":
        net.forward(s["feat"].data_ptr(), s["out"].data_ptr(), dims)
        return s["out"]
    net.forward(s["feat"].data_ptr(), s["out"].data_ptr(), dims, train=True)
    loss = net.backward(s["target"].data_ptr(), s["active"].data_ptr(), dims)
    return {"out": s["out"], "loss": float(loss), "grads": net.get_grads()}


# ------------------------------------------------------------------ least work of a pass
_MACS = 27 * (16 * 32 + 32 * 32 + 32 * 32 + 32 * 1)  # multiply-adds per vertex of one forward pass


def work(case):
    kind = case["kind"]
    if kind == "batch":
        dims = _batch_dims(case)
        # read f and g in their own type, write a float64 field
        return {"bytes": sum(w * h * d * (16 if i % 2 == 0 else 24) for i, (w, h, d) in enumerate(dims)), "flops": 0}
    W, H, D = _extents(case)
    V = W * H * D
    if kind == "correct_host":
        return {"bytes": V * (24 + 4), "flops": 0}
    if kind == "correct_dev":
        return {"bytes": V * 24, "flops": 0}
    if kind == "extract":
        return {"bytes": V * (8 + 26 * 4), "flops": 0}
    if kind == "labels":
        return {"bytes": V * (8 + 7 * 4), "flops": 0}
    if kind == "agreement":
        return {"bytes": V * 16, "flops": 0}
    if kind == "features":
        return {"bytes": V * (16 + 32 + 1), "flops": 0}
    if kind == "net_forward":
        return {"bytes": V * (32 + 4), "flops": 2 * V * _MACS}
    # forward, weight gradients (as many multiply-adds), data gradients of all layers but the first
    return {"bytes": V * (32 + 4 + 4 + 1), "flops": 2 * V * (2 * _MACS + _MACS - 27 * 16 * 32)}


# ------------------------------------------------------------------ values in 64 bits
_LAYERS = ((16, 32), (32, 32), (32, 32), (32, 16))
_DIRS = ((1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (-1, 1, 0), (1, -1, 0),
         (0, 1, 1), (0, -1, -1), (-1, 0, 1), (1, 0, -1), (-1, 1, 1), (1, -1, -1))


def _params64(net):
    """The parameters as float64 device tensors: per layer weights (27, out, in) and bias (out)."""
    p = torch.from_numpy(net.get_params()).double().cuda()
    out, at = [], 0
    for cin, cout in _LAYERS:
        n = 27 * cin * cout
        out.append((p[at:at + n].reshape(27, cout, cin).clone(), p[at + n:at + n + cout].clone()))
        at += n + cout
    return out


def _forward64(x, params, dims):
    """The network in float64: zero-padded 3x3x3 convolutions, ReLU between the layers."""
    W, H, D = dims
    x = x.reshape(D, H, W, -1)
    for i, (w, b) in enumerate(params):
        p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
        y = b.reshape(1, 1, 1, -1)
        for tap in range(27):
            dx, dy, dz = tap % 3, (tap // 3) % 3, tap // 9
            y = y + p[dz:dz + D, dy:dy + H, dx:dx + W] @ w[tap].t()
        x = torch.relu(y) if i < 3 else y
    return x[..., 0].reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "features":
        s = prepare(case, seed)
        W, H, D = _extents(case)
        f, g = s["f"].reshape(D, H, W), s["g0"].reshape(D, H, W)
        bound = (f.max() - f.min()) * case["eps"]
        slopes = torch.zeros((D, H, W, 14), dtype=torch.float64, device=f.device)
        for k, (dx, dy, dz) in enumerate(_DIRS):
            x0, x1, y0, y1, z0, z1 = (max(0, -dx), W - max(0, dx), max(0, -dy), H - max(0, dy), max(0, -dz),
                                      D - max(0, dz))
            here = f[z0:z1, y0:y1, x0:x1]
            there = f[z0 + dz:z1 + dz, y0 + dy:y1 + dy, x0 + dx:x1 + dx]
            slopes[z0:z1, y0:y1, x0:x1, k] = torch.tanh((there - here) / (4.0 * bound))
        return {"error": ((g - f) / bound).clamp(-1.0, 1.0).reshape(-1), "mismatch": None,
                "slopes": slopes.reshape(-1, 14), "active": None}
    if kind == "net_forward":
        s = prepare(case, seed)
        with torch.no_grad():
            return _forward64(s["feat"].double(), _params64(s["net"]), _extents(case))
    if kind == "net_train":
        s = prepare(case, seed)
        params = _params64(s["net"])
        for w, b in params:
            w.requires_grad_(True)
            b.requires_grad_(True)
        out = _forward64(s["feat"].double(), params, _extents(case))
        wt = s["active"].double()
        loss = (wt * (torch.tanh(out) - s["target"].double()) ** 2).sum() / wt.sum()
        loss.backward()
        grads = []
        for i, (w, b) in enumerate(params):
            gw, gb = w.grad.clone(), b.grad.clone()
            grads += [gw.reshape(-1), gb]
        return {"out": out.detach(), "loss": float(loss.detach()), "grads": torch.cat(grads).cpu().numpy()}
    return None
