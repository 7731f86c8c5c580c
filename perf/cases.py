"""What a user of paddi_b200 runs, as measurable cases.

Every case goes through the public Python API (``paddi_b200.Context`` and its
methods) on seeded series of ``paddi_b200.datagen``.  The sizes are those of
the configurations in ``paddi_b200/configs.py``, ``bench.py`` and the tests,
or generic ones of the same ranges.

``listed()`` gives the fixed cases, ``draw(rng)`` another one of their
ranges, ``prepare`` what a program holds before the call, ``run`` one call,
``work`` what the call cannot do without and ``exact`` its values in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import paddi_b200 as paddi
from paddi_b200 import datagen

POLICIES = {"merlin": paddi.R_MERLIN, "learned": paddi.R_LEARNED, "bound": paddi.R_BOUND}
KERNELS = {"auto": paddi.DIST_AUTO, "fp32": paddi.DIST_FP32, "bf16": paddi.DIST_SPLIT_BF16,
           "fp16": paddi.DIST_SPLIT_FP16}
NO_DIST = -float(np.finfo(np.float32).max)


def listed():
    return [
        # one fixed-length search of a short recording: a monitoring program calls
        # this for every new piece of data, so latency is what it sees
        {"name": "pd3_short", "kind": "pd3", "n": 4001, "m": 50, "top_k": 1, "segment": 0,
         "dist": "auto"},
        # the reference's fixed-length configuration: 4096-row segments, top-4
        {"name": "pd3_fixed", "kind": "pd3", "n": 131072, "m": 128, "top_k": 4, "segment": 4096,
         "dist": "auto"},
        # one length of a long recording
        {"name": "pd3_long_series", "kind": "pd3", "n": 1500007, "m": 300, "top_k": 1,
         "segment": 0, "dist": "auto"},
        # the drop-in for the reference's do_PD3: device buffers in, flags and nn
        # distances of all windows out
        {"name": "do_pd3_device", "kind": "do_pd3", "n": 300007, "m": 200, "r2_per_m": 0.5},
        # all options at their defaults: the reference's r schedule, host series
        {"name": "palmad_merlin", "kind": "palmad", "n": 262144, "minL": 64, "maxL": 95,
         "policy": "merlin", "dist": "auto", "series": "noise", "device": False},
        # the headline run: learned r, the whole range of lengths
        {"name": "palmad_headline", "kind": "palmad", "n": 2097152, "minL": 64, "maxL": 512,
         "policy": "learned", "dist": "auto", "series": "mixed", "device": False},
        # split-BF16 operands, the bound policy, a series already on the GPU, odd size
        {"name": "palmad_bf16_device", "kind": "palmad", "n": 524305, "minL": 100, "maxL": 131,
         "policy": "bound", "dist": "bf16", "series": "mixed", "device": True},
        # long windows: across the tensor cores' longest length into the FP32 refine
        {"name": "palmad_long_windows", "kind": "palmad", "n": 131072, "minL": 718, "maxL": 741,
         "policy": "learned", "dist": "auto", "series": "mixed", "device": False},
        # a physiological recording (quasi-periodic beats), the large configuration's
        # series and first lengths at a sixteenth of its points
        {"name": "palmad_ecg", "kind": "palmad", "n": 8388608, "minL": 128, "maxL": 139,
         "policy": "learned", "dist": "auto", "series": "ecg", "device": False},
        # many uneven series at once on four streams
        {"name": "batched_uneven", "kind": "batched", "count": 32, "min_log2": 14,
         "max_log2": 17, "minL": 32, "maxL": 55, "policy": "learned", "streams": 4},
        # the drop-in for the reference's compute_statistics
        {"name": "statistics", "kind": "stats", "n": 2097152, "m": 256},
        # training the r predictor on collected samples (forward, backward, Adam)
        {"name": "model_train", "kind": "train", "samples": 65536, "epochs": 2, "batch": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pd3", "pd3", "do_pd3", "palmad", "palmad", "palmad", "batched", "stats",
                       "train"])
    if kind == "pd3":
        n = _log_int(rng, 4000, 1500000)
        m = _log_int(rng, 32, min(700, n // 40))
        return {"kind": kind, "n": n, "m": m, "top_k": rng.choice([1, 1, 2, 4]),
                "segment": rng.choice([0, 0, 512, 4096]), "dist": rng.choice(["auto", "auto", "bf16"])}
    if kind == "do_pd3":
        return {"kind": kind, "n": _log_int(rng, 8000, 300007), "m": _log_int(rng, 32, 400),
                "r2_per_m": round(rng.uniform(0.4, 1.0), 3)}
    if kind == "palmad":
        n = _log_int(rng, 12000, 2097152)
        lo = _log_int(rng, 48, 720)
        count = _log_int(rng, 4, 64)
        policy = rng.choice(["merlin", "learned", "learned", "bound"])
        series = "noise" if policy == "merlin" else rng.choice(["noise", "mixed", "ecg"])
        if n < 40 * (lo + count):
            n = 40 * (lo + count) + rng.randrange(1000)
        if lo + count > 720:  # the FP32 refine: an order of magnitude more work per length
            n = min(n, 140000)
        return {"kind": kind, "n": n, "minL": lo, "maxL": lo + count - 1, "policy": policy,
                "dist": rng.choice(["auto", "auto", "bf16"]), "series": series,
                "device": rng.choice([False, True])}
    if kind == "batched":
        lo = _log_int(rng, 32, 128)
        return {"kind": kind, "count": rng.randrange(4, 33), "min_log2": 14,
                "max_log2": rng.choice([15, 16, 17]), "minL": lo,
                "maxL": lo + rng.randrange(4, 25), "policy": rng.choice(["learned", "bound"]),
                "streams": rng.choice([2, 4])}
    if kind == "stats":
        return {"kind": kind, "n": _log_int(rng, 5000, 4000000), "m": _log_int(rng, 16, 1024)}
    return {"kind": kind, "samples": _log_int(rng, 3000, 65536), "epochs": rng.randrange(1, 3),
            "batch": rng.choice([1024, 2048, 4096])}


# ------------------------------------------------------------------ inputs
def _series(case, seed, maxL):
    n = case["n"]
    name = case.get("series", "noise")
    if name == "ecg":
        return datagen.ecg_series(n=n, seed=seed, n_altered=max(4, n // 131072))[0]
    # anomalies as long as the longest window at most, a few per series
    hi = min(maxL, n // 32)
    kinds = ("noise", "flat", "reverse") if name == "mixed" else ("noise",)
    return datagen.palmad_series(n=n, seed=seed, n_anom=16 if n >= 1 << 17 else 6,
                                 min_len=max(hi // 4, 8), max_len=hi, kinds_cycle=kinds)[0]


def _samples(count, seed):
    """Feature rows and targets of the r predictor's shape and ranges."""
    rng = np.random.default_rng(seed)
    X = np.empty((count, paddi.MODEL_NFEAT), np.float32)
    X[:, 0] = rng.uniform(64, 1024, count) / 1024.0
    X[:, 1] = -np.abs(rng.normal(0.8, 0.4, count))
    X[:, 2:5] = rng.normal(0.01, 0.02, (count, 3))
    X[:, 5] = rng.normal(0.01, 0.02, count)
    X[:, 6] = rng.random(count) < 0.1
    X[:, 7] = rng.integers(0, 4, count) / 10.0
    X[:, 8] = rng.normal(-0.02, 0.02, count)
    X[:, 9] = np.abs(rng.normal(0, 1e-3, count))
    X[:, 10] = rng.normal(-5, 1, count)
    X[:, 11] = rng.normal(0.01, 0.01, count)
    Y = (0.6 * X[:, 5] + 0.3 * X[:, 2] + 0.1 * X[:, 11]
         + rng.normal(0, 0.01, count)).astype(np.float32)
    return X, Y


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("pd3", "do_pd3"):
        m, n = case["m"], case["n"]
        k = max(4, 2 * case.get("top_k", 1))
        x = datagen.pd3_series(n=n, seed=seed, n_anom=k, anom_len=min(max(m, 100), n // 40))[0]
        ctx = paddi.Context(device=0, distance_kernel=KERNELS[case.get("dist", "auto")])
        ctx.reserve(n, m)
        st = {"case": case, "ctx": ctx, "x": x}
        if kind == "do_pd3":
            st["d_x"] = torch.from_numpy(x).cuda()
            st["flags"] = torch.empty(n - m + 1, dtype=torch.int32, device="cuda")
            st["nn"] = torch.empty(n - m + 1, dtype=torch.float32, device="cuda")
        return st
    if kind == "palmad":
        x = _series(case, seed, case["maxL"])
        ctx = paddi.Context(device=0, distance_kernel=KERNELS[case["dist"]],
                            r_policy=POLICIES[case["policy"]])
        ctx.reserve(case["n"], case["maxL"])
        st = {"case": case, "ctx": ctx, "x": x}
        if case["device"]:
            st["d_x"] = torch.from_numpy(x).cuda()
        return st
    if kind == "batched":
        series = [s for s, _ in datagen.batch_series(case["count"], seed=seed,
                                                     min_log2=case["min_log2"],
                                                     max_log2=case["max_log2"])]
        ctx = paddi.Context(device=0, r_policy=POLICIES[case["policy"]])
        return {"case": case, "ctx": ctx, "series": series}
    if kind == "stats":
        n, m = case["n"], case["m"]
        x = datagen.random_walk_sine(n, np.random.default_rng(seed)).astype(np.float32)
        ctx = paddi.Context(device=0)
        ctx.reserve(n, m)
        return {"case": case, "ctx": ctx, "d_x": torch.from_numpy(x).cuda(),
                "mean": torch.empty(n - m + 1, dtype=torch.float32, device="cuda"),
                "std": torch.empty(n - m + 1, dtype=torch.float32, device="cuda")}
    X, Y = _samples(case["samples"], seed)
    return {"case": case, "ctx": paddi.Context(device=0), "X": X, "Y": Y,
            "init": paddi.init_params(seed)}


# ------------------------------------------------------------------ one pass
def _discords(d):
    return {"ind": np.array([q.ind for q in d], np.int64),
            "dist": np.array([q.dist for q in d], np.float32)}


def _search(d, log, lengths):
    """The discords, and per length its attempts and the last one's threshold and
    counts (the reference's times table)."""
    last = {a["m"]: a for a in log}
    tries = {m: 0 for m in lengths}
    for a in log:
        tries[a["m"]] += 1
    return {**_discords(d),
            "attempts": np.array([tries[m] for m in lengths], np.int64),
            "n_cand": np.array([last[m]["n_cand"] for m in lengths], np.int64),
            "n_disc": np.array([last[m]["n_disc"] for m in lengths], np.int64),
            "r": np.array([last[m]["r"] for m in lengths], np.float32)}


def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "pd3":
        d, log = ctx.pd3(st["x"], case["m"], top_k=case["top_k"], segment_len=case["segment"])
        return _search(d, log, [case["m"]])
    if kind == "do_pd3":
        nc = ctx.do_pd3(st["d_x"].data_ptr(), case["n"], case["m"], case["r2_per_m"] * case["m"],
                        st["flags"].data_ptr(), st["nn"].data_ptr(),
                        torch.cuda.current_stream().cuda_stream)
        return {"n_cand": nc, "flags": st["flags"], "nn": st["nn"]}
    if kind == "palmad":
        if case["device"]:
            d, log = ctx.palmad_device(st["d_x"].data_ptr(), case["n"], case["minL"],
                                       case["maxL"])
        else:
            d, log = ctx.palmad(st["x"], case["minL"], case["maxL"])
        return _search(d, log, range(case["minL"], case["maxL"] + 1))
    if kind == "batched":
        res, att = ctx.palmad_batched(st["series"], case["minL"], case["maxL"],
                                      streams=case["streams"])
        return {**_discords([q for d in res for q in d]), "attempts": np.array(att, np.int64)}
    if kind == "stats":
        ctx.compute_statistics(st["d_x"].data_ptr(), st["mean"].data_ptr(), st["std"].data_ptr(),
                               case["n"], case["m"], torch.cuda.current_stream().cuda_stream)
        return {"mean": st["mean"], "std": st["std"]}
    p, loss = ctx.model_train(st["X"], st["Y"], tau=0.1, epochs=case["epochs"],
                              batch=case["batch"], lr=3e-3, seed=1, init=st["init"])
    return {"params": p, "loss": loss}


# ------------------------------------------------------------------ the least work
def _search_work(n, m):
    """One length: the window statistics (about 10 FLOP a window), one pair test a
    window (8 FLOP; a window that is no discord needs one close neighbour) and
    the top window's distance to every other window (2 m FLOP each)."""
    N = n - m + 1
    return N * (10 + 8 + 2 * m)


def work(case):
    kind = case["kind"]
    if kind == "pd3":
        return {"bytes": 4 * case["n"], "flops": _search_work(case["n"], case["m"])}
    if kind == "do_pd3":
        N = case["n"] - case["m"] + 1
        return {"bytes": 4 * case["n"] + 8 * N, "flops": _search_work(case["n"], case["m"])}
    if kind == "palmad":
        L = range(case["minL"], case["maxL"] + 1)
        return {"bytes": 4 * case["n"] + 8 * len(L),
                "flops": sum(_search_work(case["n"], m) for m in L)}
    if kind == "batched":
        L = range(case["minL"], case["maxL"] + 1)
        n = ((1 << case["min_log2"]) + (1 << case["max_log2"])) // 2
        return {"bytes": case["count"] * (4 * n + 8 * len(L)),
                "flops": case["count"] * sum(_search_work(n, m) for m in L)}
    if kind == "stats":
        N = case["n"] - case["m"] + 1
        return {"bytes": 4 * case["n"] + 8 * N, "flops": 10 * N}
    per = 12 * 64 + 64 * 64 + 64
    return {"bytes": case["samples"] * 13 * 4 + 2 * 4 * paddi.MODEL_NPARAM,
            "flops": 6 * per * case["samples"] * case["epochs"]}


# ------------------------------------------------------------------ 64-bit values
def _nn_profile(x, m):
    """nn[i] = min over |i - j| >= m-1 of 2m (1 - rho(i, j)), FP64 on the GPU; flat
    windows have rho 0 with any other window and 1 with one another."""
    X = torch.as_tensor(x, dtype=torch.float64, device="cuda").unfold(0, m, 1)
    N = X.shape[0]
    Z = X - X.mean(1, keepdim=True)
    flat = (X == X[:, :1]).all(1)
    Z[flat] = 0.0
    nrm = Z.norm(dim=1, keepdim=True)
    Z /= torch.where(nrm > 0, nrm, torch.ones_like(nrm))
    nn = torch.empty(N, dtype=torch.float64, device="cuda")
    idx = torch.arange(N, device="cuda")
    step = max(1, min(N, (1 << 27) // N))
    for a in range(0, N, step):
        b = min(N, a + step)
        rho = Z[a:b] @ Z.T
        fa = flat[a:b]
        if bool(fa.any()):
            rho[fa] = flat.to(torch.float64)
        # the columns within m-2 of the block's rows
        lo, hi = max(0, a - m + 2), min(N, b + m - 2)
        near = (idx[a:b, None] - idx[None, lo:hi]).abs() < m - 1
        rho[:, lo:hi].masked_fill_(near, -math.inf)
        nn[a:b] = (2.0 * m * (1.0 - rho.amax(1))).clamp_min(0.0)
    return nn


def _exact_train(case, seed):
    """The same shuffles, loss and optimiser, parameters in 64 bits."""
    X, Y = _samples(case["samples"], seed)
    n, batch = len(Y), case["batch"]
    p = torch.tensor(paddi.init_params(seed), dtype=torch.float64)
    Xt, Yt = torch.tensor(X, dtype=torch.float64), torch.tensor(Y, dtype=torch.float64)
    tau, lr = float(np.float32(0.1)), float(np.float32(3e-3))
    M, V = torch.zeros_like(p), torch.zeros_like(p)
    mask = (1 << 64) - 1
    mul, add = 6364136223846793005, 1442695040888963407
    state = (1 * mul + add) & mask
    perm = list(range(n))
    t, losses = 0, []
    F, H = paddi.MODEL_NFEAT, 64
    for _ in range(case["epochs"]):
        for i in range(n - 1, 0, -1):
            state = (state * mul + add) & mask
            k = (state >> 33) % (i + 1)
            perm[i], perm[k] = perm[k], perm[i]
        order = torch.tensor(perm)
        total, nb = 0.0, 0
        for a in range(0, n, batch):
            q = order[a:a + batch]
            w = p.clone().requires_grad_(True)
            o = 0
            W1 = w[o:o + H * F].view(H, F)
            o += H * F
            b1 = w[o:o + H]
            o += H
            W2 = w[o:o + H * H].view(H, H)
            o += H * H
            b2 = w[o:o + H]
            o += H
            W3 = w[o:o + H]
            b3 = w[o + H]
            h = torch.nn.functional.gelu(Xt[q] @ W1.T + b1)
            h = torch.nn.functional.gelu(h @ W2.T + b2)
            e = Yt[q] - (h @ W3 + b3)
            loss = torch.where(e > 0, tau * e, (tau - 1.0) * e).mean()
            loss.backward()
            t += 1
            M = 0.9 * M + 0.1 * w.grad
            V = 0.999 * V + 0.001 * w.grad ** 2
            p = p - lr * (M / (1 - 0.9 ** t)) / ((V / (1 - 0.999 ** t)).sqrt() + 1e-8)
            total += float(loss.detach())
            nb += 1
        losses.append(total / nb)
    return {"params": p.numpy(), "loss": np.array(losses)}


def exact(case, seed):
    """The distances, flags, statistics and parameters in 64 bits; None where an
    all-pairs computation would take too long (2 m N^2 FLOP a length)."""
    kind = case["kind"]
    limit = 4e14
    if kind in ("pd3", "do_pd3"):
        n, m = case["n"], case["m"]
        if 2.0 * m * n * n > limit:
            return None
        k = max(4, 2 * case.get("top_k", 1))
        x = datagen.pd3_series(n=n, seed=seed, n_anom=k, anom_len=min(max(m, 100), n // 40))[0]
        nn = _nn_profile(x, m)
        if kind == "do_pd3":
            r2 = float(np.float32(case["r2_per_m"] * m))
            keep = nn >= r2
            return {"n_cand": None, "flags": None,
                    "nn": torch.where(keep, nn, torch.full_like(nn, NO_DIST))}
        picks, cur = [], nn.clone()
        for _ in range(case["top_k"]):
            j = int(cur.argmax())
            picks.append(float(nn[j]))
            cur[max(0, j - m + 2):j + m - 1] = -1.0
        return {"ind": None, "dist": np.array(picks), "attempts": None, "n_cand": None,
                "n_disc": None, "r": None}
    if kind == "palmad":
        L = range(case["minL"], case["maxL"] + 1)
        if sum(2.0 * m * case["n"] ** 2 for m in L) > limit:
            return None
        x = _series(case, seed, case["maxL"])
        return {"ind": None, "dist": np.array([float(_nn_profile(x, m).max()) for m in L]),
                "attempts": None, "n_cand": None, "n_disc": None, "r": None}
    if kind == "stats":
        n, m = case["n"], case["m"]
        x = datagen.random_walk_sine(n, np.random.default_rng(seed)).astype(np.float32)
        X = torch.as_tensor(x, dtype=torch.float64, device="cuda").unfold(0, m, 1)
        mean, std = [], []
        step = max(1, (1 << 26) // m)
        for a in range(0, X.shape[0], step):
            w = X[a:a + step]
            mean.append(w.mean(1))
            std.append(w.std(1, correction=0))
        return {"mean": torch.cat(mean), "std": torch.cat(std)}
    if kind == "train":
        return _exact_train(case, seed)
    return None
