"""Performance cases of the localization engine: the calls that a program
analysing single-molecule stacks makes, through the package's public entry
points.

A case names the call ("call"), the stack it works on and the options that
matter. Stacks are the seeded synthetic frames of localizer_b200.synth's
workloads (background plus point-sampled Gaussians, Poisson and read noise),
candidates are the package's own GLRT + adjacent-8 finder's, with the ROI
half-width of each candidate drawn from the workload's set or left to the
reference rule ceil(4 w0) (half_width 0).

``listed`` gives the named cases, ``draw`` more of the same ranges: frames of
48 to 512 pixels a side, square or not, odd sides among them; one frame to
several thousand; every fit method (0, 1, 5, 7 and the MLEwG method 6), FP32
and FP64 solves, host and device buffers; every camera storage type in both
orders.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import localizer_b200 as L
from localizer_b200 import proposal as prop

PFA = 30.0   # GLRT insensitivity of the benchmark and the tests

# mean solver iterations and algorithmic FLOPs per ROI pixel and iteration
# (model, analytic Jacobian and normal equations) of each method
ITERS = {0: 10.0, 1: 8.0, 5: 9.0, 7: 9.0}
FLOP_PX = {0: 58, 1: 46, 5: 115, 7: 115}
NPAR = {0: 5, 1: 4, 5: 7, 7: 7}


def _stack(frames, rows, cols, per_frame, **kw):
    """Plain fields of a stack: frames of cols x rows pixels with a mean of
    per_frame emitters (drawn uniformly in +-spread of it)."""
    c = dict(frames=frames, rows=rows, cols=cols, per_frame=per_frame, spread=0.0, sigma_lo=1.0, sigma_hi=2.0,
             round=False, amp=800.0, amp_logsd=0.5, bg_lo=50.0, bg_hi=200.0, pairs=0.0, w0=1.5)
    c.update(kw)
    return c


def listed():
    return [
        # one camera frame through the host-buffer call, as the reference's
        # fit_positions is called frame by frame (the call a viewer makes)
        dict(name="frame_host", call="fit_host", method=7, half=0, fp64=False,
             **_stack(1, 256, 256, 100)),
        # a live acquisition: the last few small frames, already on the GPU
        dict(name="frames_live", call="fit", method=0, half=4, fp64=False, bound=True,
             **_stack(4, 128, 128, 50, sigma_lo=1.3, sigma_hi=1.3, round=True, amp=500.0, bg_lo=100.0, bg_hi=100.0,
                      w0=1.3)),
        # the plain-method benchmark: 512 frames of 128 x 128, 9 x 9 ROIs
        dict(name="fit_small", call="fit", method=0, half=4, fp64=False, bound=True,
             **_stack(512, 128, 128, 50, sigma_lo=1.3, sigma_hi=1.3, round=True, amp=500.0, bg_lo=100.0,
                      bg_hi=100.0, w0=1.3)),
        # the batched uneven benchmark: ellipsoidal fits, mixed ROI sizes
        dict(name="fit_uneven", call="fit", method=7, half=-1, fp64=False, bound=True,
             **_stack(2000, 256, 256, 210, spread=0.9)),
        # the precision benchmark's all-FP64 arm: dim emitters, close pairs
        dict(name="fit_stress_fp64", call="fit", method=0, half=5, fp64=True, bound=True,
             **_stack(500, 256, 256, 50, sigma_lo=1.5, sigma_hi=1.5, round=True, amp=0.0, bg_lo=150.0, bg_hi=150.0,
                      pairs=0.1)),
        # the dense benchmark, symmetric fits
        dict(name="fit_dense_sym", call="fit", method=0, half=-1, fp64=False, bound=True,
             **_stack(1000, 512, 512, 650, spread=0.54)),
        # the dense benchmark, ellipsoidal fits: the largest case
        dict(name="fit_dense_ell", call="fit", method=7, half=-1, fp64=False, bound=True,
             **_stack(1000, 512, 512, 650, spread=0.54)),
        # fixed-width fits of an odd-sided camera region, default options
        # (the reference's ROI rule, no half-width promise)
        dict(name="fit_odd_fixed", call="fit", method=1, half=0, fp64=False, bound=False,
             **_stack(301, 217, 301, 120, spread=0.5, sigma_lo=1.2, sigma_hi=1.2, round=True, w0=1.2)),
        # maximum-likelihood fits of a short stack
        dict(name="mlewg", call="fit", method=6, half=-1, fp64=False, bound=True,
             **_stack(100, 256, 256, 210, spread=0.9)),
        # candidate search in the dense benchmark's frames
        dict(name="find", call="find", **_stack(500, 512, 512, 650, spread=0.54)),
        # row-major float32 camera frames into the uint16 stack
        dict(name="ingest", call="ingest", dtype="float32", row_major=True, frames=500, rows=512, cols=512),
        # one batch of the start-proposal network's training: forward and backward
        dict(name="train_batch", call="train", method=7, windows=4096),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    call = rng.choices(["fit", "fit_host", "mlewg", "find", "ingest", "train"], [10, 3, 2, 3, 2, 1])[0]
    if call == "train":
        return dict(call="train", method=rng.choice([0, 1, 5, 7]), windows=int(_log(rng, 200, 8200)))
    rows, cols = int(_log(rng, 48, 513)), int(_log(rng, 48, 513))
    if rng.random() < 0.4:
        cols = rows
    if call == "ingest":
        frames = int(_log(rng, 1, max(2, min(2000, (1 << 26) // (rows * cols)))))
        return dict(call="ingest", dtype=rng.choice(sorted(L.STORAGE_FORMATS)), row_major=rng.random() < 0.5,
                    frames=frames, rows=rows, cols=cols)
    density = _log(rng, 0.0004, 0.0031)
    most = (1 << 26) // (rows * cols)                       # a quarter of the largest listed stack
    most = min(most, int((8000 if call == "mlewg" else 150000) / max(density * rows * cols, 1.0)))
    if call == "fit_host":
        most = min(most, 300)
    frames = int(_log(rng, 1, max(2, most)))
    shaped = rng.random() < 0.5
    s = _stack(frames, rows, cols, max(3, int(density * rows * cols)), spread=rng.choice([0.0, 0.5, 0.9]),
               w0=round(rng.uniform(1.0, 1.7), 2), round=shaped, amp=rng.choice([500.0, 800.0, 0.0]),
               bg_lo=round(rng.uniform(20, 100), 1), bg_hi=round(rng.uniform(100, 250), 1),
               pairs=rng.choice([0.0, 0.0, 0.1]))
    if call == "find":
        return dict(call="find", **s)
    half = rng.choice([0, -1, rng.randint(2, 8)])
    if call == "mlewg":
        return dict(call="fit", method=6, half=half, fp64=False, bound=rng.random() < 0.5, **s)
    method = rng.choice([0, 0, 1, 5, 7, 7])
    if call == "fit_host":
        return dict(call="fit_host", method=method, half=half, fp64=False, **s)
    return dict(call="fit", method=method, half=half, fp64=frames * s["per_frame"] < 20000 and rng.random() < 0.3,
                bound=rng.random() < 0.5, **s)


# ---------------------------------------------------------------- inputs --

def _frames(case, seed):
    """The case's stack on the GPU: int16 tensor (frames, cols, rows) holding
    uint16 counts, rendered by the package's workload generator."""
    rng = np.random.default_rng([seed, 11])
    n, rows, cols = case["frames"], case["rows"], case["cols"]
    mean = case["per_frame"]
    lo, hi = int(mean * (1 - case["spread"])), int(mean * (1 + case["spread"]))
    counts = rng.integers(max(lo, 1), max(hi, 1) + 1, size=n)
    k = int(counts.sum())
    frame = np.repeat(np.arange(n), counts)
    x, y = rng.uniform(5, rows - 6, k), rng.uniform(5, cols - 6, k)
    if case["pairs"] > 0:
        at = np.nonzero(rng.random(k) < case["pairs"])[0]
        at = at[at > 0]
        at = at[frame[at] == frame[at - 1]]
        d, ang = rng.uniform(1.5, 3.0, at.size), rng.uniform(0, 2 * np.pi, at.size)
        x[at] = np.clip(x[at - 1] + d * np.cos(ang), 5, rows - 6)
        y[at] = np.clip(y[at - 1] + d * np.sin(ang), 5, cols - 6)
    # amplitude 0: the dim workload, uniform 50 to 200 photons
    amp = rng.uniform(50, 200, k) if case["amp"] == 0 else \
        np.exp(np.log(case["amp"]) + case["amp_logsd"] * rng.standard_normal(k))
    sx = rng.uniform(case["sigma_lo"], case["sigma_hi"], k)
    sy = sx if case["round"] else rng.uniform(case["sigma_lo"], case["sigma_hi"], k)
    bg = torch.from_numpy(rng.uniform(case["bg_lo"], case["bg_hi"], n).astype(np.float32)).cuda()
    em = torch.from_numpy(np.stack([x, y, amp, sx, sy], axis=1).astype(np.float32)).cuda()
    start = torch.from_numpy(np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)).cuda()
    out = torch.empty((n, cols, rows), dtype=torch.int16, device="cuda")
    if L.lib().loc_synth_frames(out.data_ptr(), n, rows, cols, em.data_ptr(), start.data_ptr(), bg.data_ptr(), 2.0,
                                seed, 0) != 0:
        raise RuntimeError("loc_synth_frames failed")
    torch.cuda.synchronize()
    return out


def _n_cands(case):
    return max(1, int(0.8 * case["frames"] * case["per_frame"]))


def _candidates(case, frames, seed):
    raw, _ = L.find_candidates_device(frames, PFA, case["w0"])
    c = raw.cpu().numpy().view(L.CANDIDATE_DTYPE).copy()
    # as many as the case says, whatever the seed: part of what was found, or
    # some of it twice (a case's outputs have one shape)
    n = _n_cands(case)
    if len(c) == 0:
        c = np.zeros(1, dtype=L.CANDIDATE_DTYPE)
        c["x"], c["y"], c["intensity"], c["background"] = case["rows"] // 2, case["cols"] // 2, 100.0, case["bg_lo"]
    at = np.random.default_rng([seed, 13]).permutation(max(len(c), n))[:n] % len(c)
    c = c[np.sort(at)]
    if case["half"] > 0:
        c["half_width"] = case["half"]
    elif case["half"] < 0:   # mixed ROI sizes
        c["half_width"] = np.random.default_rng([seed, 17]).choice(np.array([3, 4, 5, 6]), size=len(c))
    return c


def prepare(case, seed):
    call = case["call"]
    if call == "ingest":
        g = torch.Generator(device="cuda").manual_seed(seed)
        shape = (case["frames"], case["rows"], case["cols"]) if case["row_major"] else \
            (case["frames"], case["cols"], case["rows"])
        dtype = getattr(torch, case["dtype"])
        hi = 127 if case["dtype"] == "int8" else 255 if case["dtype"] == "uint8" else 4095
        counts = torch.randint(0, hi + 1, shape, generator=g, device="cuda", dtype=torch.int32)
        return dict(case=case, src=counts.to(dtype))
    if call == "train":
        rois, truth = prop.synth_rois(case["windows"], case["method"] in (5, 7), seed, truth=True)
        x, y, a, sx, sy, b = truth.unbind(1)
        zero = torch.zeros_like(a)
        p = prop.NOUT[case["method"]]
        cols = {4: [a, x - 5, y - 5, b], 5: [a, sx, x - 5, y - 5, b], 7: [a, sx, sy, x - 5, y - 5, zero, b]}[p]
        lam = {4: [40, 6, 6, 17], 5: [38, 38, 6, 6, 17], 7: [42, 14, 14, 3.5, 3.5, 49, 16]}[p]
        net = prop.Proposal(case["method"], 0, seed)
        return dict(case=case, net=net, rois=rois, labels=torch.stack(cols, 1).contiguous(),
                    lam=np.array(lam, dtype=np.float32))
    frames = _frames(case, seed)
    if call == "find":
        # the analysis keeps its candidate list in a buffer of its own
        room = 40 * (3 * case["frames"] * case["per_frame"] + 1024)
        return dict(case=case, frames=frames, found=torch.zeros(room, dtype=torch.uint8, device="cuda"))
    cands = _candidates(case, frames, seed)
    if call == "fit_host":
        return dict(case=case, eng=L.default_engine(), frames=frames.cpu().numpy().view(np.uint16), cands=cands)
    n, ncol = len(cands), L.lib().loc_output_columns(case["method"])
    opts = L.default_options(precision=int(case["fp64"]))
    if case["bound"]:
        r_default = math.ceil(4 * case["w0"])
        opts.max_half_width = int(np.where(cands["half_width"] > 0, cands["half_width"], r_default).max()) if n else 1
    return dict(case=case, eng=L.default_engine(), frames=frames, n=n, opts=opts,
                cands=torch.from_numpy(cands.view(np.uint8)).cuda() if n else torch.empty(40, dtype=torch.uint8,
                                                                                          device="cuda"),
                out=torch.zeros((n, ncol), dtype=torch.float64, device="cuda"),
                flags=torch.zeros(n, dtype=torch.uint8, device="cuda"))


# ------------------------------------------------------------------ calls --

def run(state):
    case = state["case"]
    call = case["call"]
    if call == "fit":
        f = state["frames"]
        state["eng"].fit_device(f.data_ptr(), f.shape[0], f.shape[2], f.shape[1], state["cands"].data_ptr(),
                                state["n"], case["method"], case["w0"], 1.0, state["out"].data_ptr(),
                                state["flags"].data_ptr(), torch.cuda.current_stream().cuda_stream, state["opts"])
        return {"rows": state["out"], "flags": state["flags"]}
    if call == "fit_host":
        rows, flags = state["eng"].fit_host(state["frames"], state["cands"], case["method"], case["w0"])
        return {"rows": rows, "flags": flags}
    if call == "find":
        cands, n = L.find_candidates_device(state["frames"], PFA, case["w0"],
                                            torch.cuda.current_stream().cuda_stream)
        found = state["found"]
        found[:len(cands)].copy_(cands)
        found[len(cands):].zero_()
        return {"candidates": found, "n": n}
    if call == "ingest":
        stack, changed = L.ingest_frames(state["src"], case["row_major"], torch.cuda.current_stream().cuda_stream)
        return {"stack": stack, "changed": changed}
    grad, loss = state["net"].gradient(state["rois"], state["labels"], state["lam"],
                                       stream=torch.cuda.current_stream().cuda_stream)
    return {"gradient": grad, "loss": loss}


def work(case):
    call = case["call"]
    if call == "train":
        n = case["windows"]
        p = prop.NOUT[case["method"]]
        weights = 14048 + 801 * p
        # forward 0.91 MFLOP a window, backward twice that
        return {"bytes": n * (242 + 4 * p) + 8 * weights, "flops": n * 2.8e6}
    px = case["frames"] * case["rows"] * case["cols"]
    if call == "ingest":
        return {"bytes": px * (2 + torch.empty(0, dtype=getattr(torch, case["dtype"])).element_size()), "flops": 0}
    n = _n_cands(case)
    if call == "find":
        ws = math.ceil(4 * case["w0"]) | 1
        return {"bytes": 2 * px + 40 * n, "flops": 2 * ws * ws * px}
    m = case["method"]
    half = [case["half"]] if case["half"] > 0 else [math.ceil(4 * case["w0"])] if case["half"] == 0 else [3, 4, 5, 6]
    roi = sum((2 * h + 1) ** 2 for h in half) / len(half)
    ncol = {0: 14, 1: 12, 5: 18, 6: 10, 7: 18}[m]
    traffic = n * (2 * roi + 40 + 8 * ncol + 1)
    if call == "fit_host":
        traffic += 2 * px
    if m == 6:   # 200 simplex iterations of about 1.7 objective evaluations, 20 operations a pixel
        return {"bytes": traffic, "flops": n * 340 * roi * 20}
    p = NPAR[m]
    return {"bytes": traffic, "flops": n * ITERS[m] * (FLOP_PX[m] * roi + p ** 3 / 3 + 2 * p * p)}


# ------------------------------------------------------------------ exact --

def exact(case, seed):
    """The training batch in 64 bits. The other outputs have no such value:
    candidates, flags and ingested counts are whole numbers and bytes, and a
    fit's row is where its iteration path ends under a loose stopping test,
    which only the algorithm itself defines (the rows of the start are the
    yardstick there)."""
    if case["call"] != "train":
        return None
    s = prepare(case, seed)
    p = prop.NOUT[case["method"]]
    w = torch.from_numpy(s["net"].weights()).cuda().double().requires_grad_(True)
    win = (s["rois"].to(torch.int32) & 0xFFFF).double().reshape(-1, 11, 11)
    border = torch.ones(11, 11, dtype=torch.bool, device="cuda")
    border[1:-1, 1:-1] = False
    b0 = win[:, border].sum(1) / 40
    s0 = (win[:, 4:7, 4:7].reshape(-1, 9).sum(1) / 9 - b0).clamp_min(10.0)
    a = ((win - b0[:, None, None]) / s0[:, None, None])[:, None]
    conv = torch.nn.functional.conv2d
    a = torch.relu(conv(a, w[0:144].reshape(16, 1, 3, 3), w[144:160]))
    a = torch.relu(conv(a, w[160:4768].reshape(32, 16, 3, 3), w[4768:4800]))
    a = torch.relu(conv(a, w[4800:14016].reshape(32, 32, 3, 3), w[14016:14048]))
    out = a.reshape(-1, 800) @ w[14048:14048 + 800 * p].reshape(p, 800).T + w[14048 + 800 * p:14048 + 801 * p]
    cols = []
    for j, role in enumerate(prop.ROLES[p]):
        v = s["labels"][:, j].double()
        cols.append(torch.log(v.clamp_min(1.0) / s0) if role == 0 else
                    torch.log(v.clamp_min(0.05) / prop.SIGMA_REF) if role == 1 else
                    (v - b0) / s0 if role == 5 else v)
    lam = torch.from_numpy(s["lam"]).cuda().double()
    loss = (lam * (out - torch.stack(cols, 1)) ** 2).sum(1).mean()
    loss.backward()
    return {"gradient": w.grad, "loss": float(loss.detach())}
