#!/usr/bin/env python
"""Benchmark of the tensor-voting path on one GB300 per process.

Workload (default, --config c4, the surrogate study's field): a seeded
synthetic 384^3 float32 volume of 64 tubes (radius 1-3 voxels, 8-segment
piecewise-linear centrelines) plus N(0, 0.05) noise -> 3x3 structure tensor
(gradient, outer product, separable Gaussian sigma 1.5, 9 taps, same-size
output) -> TK stick + plate voting at sigma 4 (w = 25, samples = 20; the
plate is the exact orientation integral) -> per-voxel 3x3 eigendecomposition
of the voted field.  --config c2 is the same recipe at 256^3.  One "step" is
that whole pass over the volume; the metric is voxels per second.

  value     device-resident: input already in HBM, the pipeline call
            (tvgb_pipeline3) on device arrays, CUDA events on its stream,
            L2 flushed (256 MiB write) between timed steps outside the events.
  e2e       the same call with pinned HOST buffers: the host->device copy of
            the volume and the device->host copy of the voted field,
            eigenvalues and eigenvectors are inside the timed region.
  roofline  the dominant kernel (k_sep_xy, the x and y sums of the separable
            vote; k_vote3_fast where the pair-by-pair vote runs): algorithmic
            FP32 flops / its duration (library CUDA-event timing).
  cpu_baseline  the reference's CPU algorithm (the C port in oracle/, the
            reference's own sampled plate rule) on a bounded interior sample,
            all host cores, rank 0 at N = 1 only.
  surrogate the learned plate vote against the plain 64-orientation integral
            and the exact closed form on an interior block of the same field
            (network trained first, on the GPU): voxels/s of each, their
            ratios, errors against the exact vote, the judge's recomputes.

--impl reference runs that CPU reference alone (rank 0), one bounded sample
per step.  Under torchrun every rank processes its own volume (weak scaling,
no collective on the data path); the reported time is the max over ranks.
"""
import argparse
import ctypes
import json
import os
import re
import subprocess
import sys
import tempfile
import time

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)

METRIC = "3D tensor-vote voxels/s (σ=4): surrogate vs plain, same GB300, ≤1e-3 rel err"

C2 = dict(name="C2", n=256, n_tubes=64, r_range=(1.0, 3.0), noise_sd=0.05, seed=2, n_sheets=0, sigma_st=1.5,
          sigma=4.0, w=25, samples=20, ball=False)
# the 384^3 field of the surrogate study, run here on the plain path
C4 = dict(C2, name="C4", n=384, seed=4)
# capacity: tubes and sheets, stick + plate + ball at sigma 6
C5 = dict(name="C5", n=512, n_tubes=256, r_range=(1.0, 4.0), noise_sd=0.1, seed=5, n_sheets=32, sigma_st=2.0,
          sigma=6.0, w=37, samples=20, ball=True)
CONFIGS3 = {"c2": C2, "c4": C4, "c5": C5}

# Algorithmic FP32 flops per in-bounds (receiver, voter) pair of the fast
# kernel, FMA = 2, counted from the formulas in tiralib_gb300/csrc/vote3.cu:
#   stick (power 1): q.o 2, 2ug 1, r 6, u^2 1, eta 2, term 1, term*r 3, 6 accumulations 12 = 28
#   plate (closed form): n.o 2, 2vg 1, m 6, h 6, v^2 1, cA 2, sA 1, sB 1, identity 1,
#                        sA*m 3, sB*h 3, 12 accumulations 24 = 51
FLOPS_PER_PAIR = 28 + 51
#   ball (closed form): identity 2, lb*w 1, w*o 3, 6 accumulations 12 = 18
FLOPS_PER_PAIR_BALL = 18
FP32_LANES_PER_SM = 128


def pairs_count(dims, hw, zrange=None):
    """Exact number of in-bounds (receiver, voter) pairs: product over axes of
    sum_x #{o in [-hw, hw] : 0 <= x + o < s}; zrange restricts the receivers'
    first axis to [z0, z1) (a z-slab)."""
    p = 1
    for axis, s in enumerate(dims):
        lo, hi = zrange if (axis == 0 and zrange) else (0, s)
        tot = 0
        for x in range(lo, hi):
            tot += min(s - 1, x + hw) - max(0, x - hw) + 1
        p *= tot
    return p


def fp32_peak(tv, sms, max_mhz):
    """The FP32 denominator: measured in this run by the library's FMA
    throughput kernel (independent packed-FMA chains on every SM, with the SM
    clock it ran at), beside the nominal rate at the maximum SM clock."""
    import ctypes
    tf, mhz = ctypes.c_double(0.0), ctypes.c_double(0.0)
    tv.lib().tvgb_fp32_peak(ctypes.byref(tf), ctypes.byref(mhz), None)
    nominal = sms * FP32_LANES_PER_SM * 2 * max_mhz * 1e6 / 1e12
    return {"measured": tf.value, "measured_sm_mhz": mhz.value, "nominal": nominal,
            "source": f"nominal FP32: {sms} SMs x {FP32_LANES_PER_SM} FMA lanes x 2 x {max_mhz:.0f} MHz "
                      f"(MEASURED_PEAKS.json has no FP32 figure); beside it, the rate a plain kernel of independent "
                      f"FP32 FMA chains on all SMs reached in this run (~40 ms at {mhz.value:.0f} MHz)"}


def dist_env():
    return int(os.environ.get("RANK", 0)), int(os.environ.get("WORLD_SIZE", 1)), int(os.environ.get("LOCAL_RANK", 0))


class ClockSampler:
    """nvidia-smi clock / throttle-reason sampling during the timed region."""
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.gpu_index = gpu_index
        self.proc = None
        self.path = None

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                                          "-lms", "200", "-i", str(self.gpu_index)],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *a):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        rows = []
        try:
            for line in open(self.path):
                parts = [p.strip() for p in line.split(",")]
                if len(parts) >= 9:
                    rows.append(parts)
        except Exception:
            pass
        finally:
            if self.path and os.path.exists(self.path):
                os.remove(self.path)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "", 1).isdigit()]
        smax = [float(r[2]) for r in rows if r[2].replace(".", "", 1).isdigit()]
        pw = [float(r[3]) for r in rows if r[3].replace(".", "", 1).isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for r in rows for k in range(4) if r[5 + k].lower() == "active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "power_w_max": max(pw) if pw else None, "samples": len(rows), "reasons": reasons}


def gpu_index_for(local_rank):
    vis = os.environ.get("CUDA_VISIBLE_DEVICES")
    if vis:
        items = [v.strip() for v in vis.split(",") if v.strip()]
        if local_rank < len(items) and items[local_rank].isdigit():
            return int(items[local_rank])
    return local_rank


def cpu_reference_sample(vol, cfg, block=16, seed=0, threads=None, detail=None):
    """The reference's CPU algorithm on one bounded sample: an interior
    block^3 receiver block with its window halo.  Structure tensor (oracle
    restatement of volume::gradient + gaussian_convolve3), cpu::tensorvote3's
    stick + sampled plate (samples = cfg['samples']) for the block's
    receivers, eigendecomposition of their voted tensors.  Returns (seconds,
    receivers, threads)."""
    from oracle import oracle as O
    threads = threads or os.cpu_count() or 1
    hw = cfg["w"] // 2
    K = O.lib().or_ksize3(cfg["sigma_st"])
    R = K // 2
    n = vol.shape[0]
    rng = np.random.default_rng(seed)
    pad = hw + R + 1
    z0, y0, x0 = (int(v) for v in rng.integers(pad, n - pad - block, 3))
    t0 = time.perf_counter()
    crop = vol[z0 - hw - R - 1:z0 + block + hw + R + 1, y0 - hw - R - 1:y0 + block + hw + R + 1,
               x0 - hw - R - 1:x0 + block + hw + R + 1]
    st = O.structure_tensor3(crop, cfg["sigma_st"], 0)        # valid: interior of the same-size field
    st = st[:, 1:-1, 1:-1, 1:-1]                                # drop the gradient-only rim
    s6 = np.moveaxis(st, 0, -1)
    m9 = np.ascontiguousarray(s6[..., [0, 1, 2, 1, 3, 4, 2, 4, 5]].reshape(s6.shape[:3] + (3, 3)))
    S = m9.shape[0]
    zz, yy, xx = np.meshgrid(np.arange(hw, hw + block), np.arange(hw, hw + block), np.arange(hw, hw + block),
                             indexing="ij")
    rec = ((zz * S + yy) * S + xx).ravel()
    out = O.tensorvote3_receivers(m9, rec, cfg["sigma"], 0.0, cfg["w"], 1, samples=cfg["samples"], threads=threads,
                                  is_atv=bool(cfg.get("atv")))
    voted = out.reshape(-1, 9)[rec]
    ev = O.evals3(voted)
    vec = O.evecs3cart(voted, ev)
    dt = time.perf_counter() - t0
    if detail is not None:
        detail.update(block=(z0, y0, x0, block), field=m9, receivers=rec, voted=voted, evals=ev, evecs=vec)
    return dt, rec.size, threads


def accuracy_against_cpu(detail, cfg, out_d, ev_d, vec_d, threads, precise=None):
    """The GPU pipeline's results at the CPU sample's receivers against (a)
    the reference's algorithm on the CPU (oracle port, same input volume,
    its own structure tensor) and (b) the FP64 oracle (FP64 eigenvectors of
    the voters, FP64 vote) on that structure tensor.  Voted tensors: the six
    entries eigen.h reads back; per receiver ||d|| / ||ref|| (Frobenius over
    the six), and max|d| / max|ref| over the block.  Eigenvalues: per
    receiver max|d| / max|ref|.  Eigenvectors: angle between matching
    vectors (up to sign), largest and smallest."""
    from oracle import oracle as O
    z0, y0, x0, b = detail["block"]
    sl = (slice(z0, z0 + b), slice(y0, y0 + b), slice(x0, x0 + b))
    g6 = np.moveaxis(out_d[(slice(None),) + sl].cpu().numpy(), 0, -1).reshape(-1, 6).astype(np.float64)
    gev = ev_d[sl].cpu().numpy().reshape(-1, 3).astype(np.float64)
    gvec = vec_d[sl].cpu().numpy().reshape(-1, 3, 3).astype(np.float64)
    idx6 = [0, 1, 2, 4, 5, 8]
    c6 = detail["voted"].reshape(-1, 9)[:, idx6].astype(np.float64)
    f64 = None if cfg.get("atv") else O.tensorvote3_f64(
        detail["field"], cfg["sigma"], 0.0, cfg["w"], 1, ball=cfg["ball"], receivers=detail["receivers"],
        threads=threads).reshape(-1, 6)[detail["receivers"]]
    wgt = np.array([1, 2, 2, 1, 2, 1], np.float64)   # off-diagonal entries count twice in the Frobenius norm

    def tensor_err(a, ref):
        per = np.sqrt((wgt * (a - ref) ** 2).sum(1) / np.maximum((wgt * ref ** 2).sum(1), 1e-300))
        return {"per_receiver_max": float(per.max()), "per_receiver_median": float(np.median(per)),
                "max_abs_over_max": float(np.abs(a - ref).max() / np.abs(ref).max())}

    cev = detail["evals"].astype(np.float64)
    ev_rel = np.abs(gev - cev).max(1) / np.maximum(np.abs(cev).max(1), 1e-300)
    cvec = detail["evecs"].reshape(-1, 3, 3).astype(np.float64)
    cosang = np.clip(np.abs((gvec * cvec).sum(2)), 0.0, 1.0)          # rows e0, e1, e2
    ang = np.arccos(cosang)
    out = {"receivers": int(b ** 3), "block_origin_zyx": [int(z0), int(y0), int(x0)],
           "voted_vs_reference_cpu": tensor_err(g6, c6),
           "voted_vs_fp64": tensor_err(g6, f64) if f64 is not None else None,
           "eigenvalues_vs_reference_cpu": {"max": float(ev_rel.max()), "median": float(np.median(ev_rel))},
           "eigenvector_angle_rad_vs_reference_cpu": {"e2_max": float(ang[:, 2].max()),
                                                      "e2_median": float(np.median(ang[:, 2])),
                                                      "e0_max": float(ang[:, 0].max()),
                                                      "e0_median": float(np.median(ang[:, 0]))}}
    out["note_fp64"] = ("the reference's eigen.h thresholds are absolute (1e-6 on b^2+d^2+e^2): the noise voxels' "
                        "structure tensors fall under them, so the reference's voter eigenvectors, which parity "
                        "mode reproduces, are far from FP64's; precise mode (scaled, relative thresholds, FP64 "
                        "refinement of near-degenerate pairs) is the one to judge against FP64")
    if precise is not None:
        p_out, p_ev, p_vec = precise
        p6 = np.moveaxis(p_out[(slice(None),) + sl].cpu().numpy(), 0, -1).reshape(-1, 6).astype(np.float64)
        pev = p_ev[sl].cpu().numpy().reshape(-1, 3).astype(np.float64)
        pvec = p_vec[sl].cpu().numpy().reshape(-1, 3, 3).astype(np.float64)
        fev, fvec = O.eig3_f64(f64)
        prel = np.abs(pev - fev).max(1) / np.maximum(np.abs(fev).max(1), 1e-300)
        pang = np.arccos(np.clip(np.abs((pvec * fvec).sum(2)), 0.0, 1.0))
        # the eigensolver alone: FP64 Jacobi of the GPU's own voted tensors
        sev, svec = O.eig3_f64(p6)
        srel = np.abs(pev - sev).max(1) / np.maximum(np.abs(sev).max(1), 1e-300)
        sang = np.arccos(np.clip(np.abs((pvec * svec).sum(2)), 0.0, 1.0))
        out["precise_mode"] = {
            "voted_vs_fp64": tensor_err(p6, f64),
            "eigenvalues_vs_fp64": {"max": float(prel.max()), "median": float(np.median(prel))},
            "eigenvector_angle_rad_vs_fp64": {"e2_max": float(pang[:, 2].max()),
                                              "e2_median": float(np.median(pang[:, 2])),
                                              "e0_max": float(pang[:, 0].max()),
                                              "e0_median": float(np.median(pang[:, 0]))},
            "eigensolver_alone": {"eigenvalues_max": float(srel.max()), "eigenvalues_median": float(np.median(srel)),
                                  "angle_rad_e2_max": float(sang[:, 2].max()),
                                  "angle_rad_e2_median": float(np.median(sang[:, 2])),
                                  "angle_rad_e0_max": float(sang[:, 0].max()),
                                  "angle_rad_e0_median": float(np.median(sang[:, 0]))},
            "note": "the eigenvector angles against the FP64 vote follow the voted tensors' own FP32 error divided "
                    "by their eigenvalue gaps; eigensolver_alone compares with FP64 Jacobi of the same tensors"}
    if cfg["ball"]:
        out["note_ball"] = ("the reference's CPU algorithm has no TK ball term: voted_vs_reference_cpu includes the "
                            "GPU's ball vote; the FP64 comparisons include it on both sides")
    return out


def config3(args):
    cfg = dict(CONFIGS3[args.config])
    if args.size:
        cfg["n"] = args.size
    cfg["atv"] = bool(getattr(args, "atv", False))
    return cfg


def make_volume(cfg, dev=None):
    """The config's tube (and sheet) volume: on the host below 384^3, else
    rasterised on `dev` (same geometry; device-generator noise)."""
    from tiralib_gb300 import workloads as W
    kw = dict(n_tubes=cfg["n_tubes"], r_range=cfg["r_range"], noise_sd=cfg["noise_sd"], seed=cfg["seed"],
              n_sheets=cfg["n_sheets"])
    if dev is not None and cfg["n"] >= 384:
        return W.tube_volume_device(cfg["n"], dev, **kw)
    return W.tube_volume(cfg["n"], **kw)


def metric_for(cfg):
    if cfg.get("atv"):
        return (f"3D ATV voxels/s ({cfg['name']}: analytical tensor voting, sigma={cfg['sigma']:g}, "
                f"stick+plate+ball)")
    if cfg["name"] in ("C2", "C4"):
        return METRIC
    return (f"3D tensor-vote voxels/s ({cfg['name']}: sigma={cfg['sigma']:g}, "
            f"stick+plate{'+ball' if cfg['ball'] else ''}, plain path)")


def run_reference(args, rank):
    if rank != 0:
        return
    import torch
    cfg = config3(args)
    vol = make_volume(cfg, torch.device("cuda", 0) if torch.cuda.is_available() else None)
    if not isinstance(vol, np.ndarray):
        vol = vol.cpu().numpy()
    for i in range(args.warmup):
        cpu_reference_sample(vol, cfg, block=args.ref_block, seed=1000 + i)
    times, nrec, th = [], 0, 1
    for i in range(args.steps):
        t, nrec, th = cpu_reference_sample(vol, cfg, block=args.ref_block, seed=i)
        times.append(t)
    total = float(np.sum(times))
    value = args.steps * nrec / total
    algo = ("ATV (tira::cpu::tensorvote3_atv's algorithm, tensorvote.h:710)" if cfg["atv"] else
            f"stick + {cfg['samples']}-sample plate (tira::cpu::tensorvote3's algorithm"
            f"{'; the reference has no TK ball' if cfg['ball'] else ''})")
    sample = (f"{args.ref_block}^3 interior receivers (+{cfg['w'] // 2}-voxel window halo) of the {cfg['n']}^3 "
              f"volume per step: structure tensor, {algo}, 3x3 eigen of the voted tensors; OpenMP over receivers")
    line = {
        "impl": "reference", "metric": metric_for(cfg), "value": value, "unit": "voxels/s", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * total / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": config_dict(cfg),
        "cpu_baseline": {"value": value, "unit": "voxels/s", "cores": th, "kind": "port", "sample": sample},
        "e2e": {"value": value, "unit": "voxels/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def config_dict(cfg):
    n = cfg["n"]
    terms = "stick+plate+ball" if cfg["ball"] else "stick+plate"
    sheets = f" + {cfg['n_sheets']} sheets" if cfg["n_sheets"] else ""
    vote = (f"ATV vote (tensorvote.h:710; sigma {cfg['sigma']:g}, w {cfg['w']})" if cfg.get("atv") else
            f"TK {terms} vote (sigma {cfg['sigma']:g}, w {cfg['w']}, samples {cfg['samples']})")
    return {"workload": f"{cfg['name']}: {n}^3 tube volume{sheets} -> structure tensor (sigma {cfg['sigma_st']:g}) -> "
                        f"{vote} -> fused 3x3 eigendecomposition",
            "volume": [cfg["n"]] * 3, "tubes": cfg["n_tubes"], "tube_radius": list(cfg["r_range"]),
            "sheets": cfg["n_sheets"], "noise_sd": cfg["noise_sd"], "seed": cfg["seed"],
            "sigma_structure": cfg["sigma_st"], "sigma_vote": cfg["sigma"], "window": cfg["w"],
            "samples": cfg["samples"], "power": 1, "ball": cfg["ball"], "atv": bool(cfg.get("atv")),
            "path": "plain (exact plate orientation integral, no surrogate)",
            "l2_flush": "256 MiB write between timed steps (outside the events)"}


def parse_profile(text):
    out = {}
    for line in text.strip().splitlines():
        parts = line.split()
        if len(parts) == 3:
            out[parts[0]] = (int(parts[1]), float(parts[2]))
    return out


def profiled_traffic(kernel, workload="c2", units=None):
    """DRAM traffic per launch of a kernel, as recorded in its committed ncu
    summary (profiles/<kernel>_<workload>.md), not measured in this run.  The
    summary holds `dram_bytes_per_launch: <bytes>` and `traffic_source:
    <capture, date>`; `dram_units_per_launch: <n>` when the capture ran a
    smaller case, whose traffic is then scaled by units / n (traffic grows in
    proportion to the units processed).  Returns {"traffic": bytes or None,
    "traffic_source": text or None}."""
    out = {"traffic": None, "traffic_source": None}
    path = os.path.join(HERE, "profiles", f"{kernel}_{workload}.md")
    if not os.path.exists(path):
        return out
    fields = {}
    for line in open(path):
        line = line.strip()
        for key in ("dram_bytes_per_launch", "dram_units_per_launch", "traffic_source"):
            if line.startswith(key + ":"):
                fields[key] = line.split(":", 1)[1].strip()
    try:
        t = float(fields["dram_bytes_per_launch"])
    except (KeyError, ValueError):
        return out
    src = f"profiles/{kernel}_{workload}.md: {fields.get('traffic_source', 'ncu capture')}"
    if units and "dram_units_per_launch" in fields:
        cap = float(fields["dram_units_per_launch"])
        t *= units / cap
        src += f"; scaled by {units:.4g} / {cap:.4g} units"
    out["traffic"] = t
    out["traffic_source"] = src
    return out


def separable_taps(sigma, hw):
    """Weights per axis, summed over the exponentials, of the separable vote
    at one Gaussian: sum of 2 h + 1, by the tables and the half-width rule of
    tiralib_gb300/csrc/vote3_sep.cu (sep_terms)."""
    text = open(os.path.join(HERE, "tiralib_gb300", "csrc", "vote3_sep_tables.inc")).read()
    num = r"\{([^{}]*)\}"
    for row in re.finditer(r"\{(\d+),\s*(\d+),\s*" + r",\s*".join([num] * 4), text):
        if min(3.0 * hw * hw, 104.0 * sigma ** 2) > int(row[1]):
            continue
        b, *w = [[float(v) for v in row[i].split(",") if v.strip()] for i in (3, 4, 5, 6)]
        taps = 0
        for t in range(int(row[2])):
            h = hw
            while t > 0 and h > 1:
                q = float(h * h)
                top = max(abs(w[k][t]) * q ** (k + 1) for k in range(3)) * np.exp(-b[t] * q)
                if (b[t] + sigma ** -2) * q < 104.0 and (q * b[t] < 3.0 or top > 3e-8):
                    break
                h -= 1
            taps += 2 * h + 1
        return taps
    return 0


def run_ours(args, rank, world, local_rank):
    import torch
    import ctypes
    import tiralib_gb300 as tv
    from tiralib_gb300 import workloads as W

    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    dist = None
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", device_id=dev)
    cfg = config3(args)
    vol = make_volume(cfg, dev)
    vol_np = vol if isinstance(vol, np.ndarray) else vol.cpu().numpy()
    del vol
    nvox = vol_np.size
    dims = vol_np.shape
    vol_h = torch.from_numpy(vol_np).pin_memory()
    vol_d = vol_h.to(dev)
    out_d = torch.empty((6,) + dims, device=dev)
    ev_d = torch.empty(dims + (3,), device=dev)
    vec_d = torch.empty(dims + (3, 3), device=dev)
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)
    kw = dict(sigma_st=cfg["sigma_st"], sigma1=cfg["sigma"], w=cfg["w"], samples=cfg["samples"], st_mode="same",
              out_layout="planes", evecs="cartesian", ball=cfg["ball"], is_atv=cfg["atv"])
    strong = args.split == "slabs" and world > 1
    if strong:
        # strong scaling: one volume, each rank votes its z-slab (+ halos); no collective on the data path
        from tiralib_gb300 import slabs
        z0, z1 = slabs.partition(dims[0], world)[rank]
        skw = dict(sigma_st=cfg["sigma_st"], sigma1=cfg["sigma"], w=cfg["w"], samples=cfg["samples"],
                   ball=cfg["ball"])

    def step():
        if strong:
            slabs.pipeline3_slab(vol_d, z0, z1, **skw)
        else:
            tv.pipeline3(vol_d, outputs=(out_d, ev_d, vec_d), **kw)

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    if dist:
        dist.barrier()
    stream = torch.cuda.current_stream()
    lib = tv.lib()
    torch.cuda.reset_peak_memory_stats(dev)
    tv.memory_stats(reset_peak=True)
    lib.tvgb_profile_enable(1)
    buf = ctypes.create_string_buffer(1 << 14)
    lib.tvgb_profile_read(buf, len(buf))        # clear
    l0 = tv.launch_count()
    times = []
    with ClockSampler(gpu_index_for(local_rank)) as clk:
        torch.cuda.synchronize()
        for _ in range(args.steps):
            flush.zero_()
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            step()
            e1.record(stream)
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        torch.cuda.synchronize()
    launches = tv.launch_count() - l0
    free_b, total_b = torch.cuda.mem_get_info(dev)
    memory = {"torch_tensors_peak_bytes": int(torch.cuda.max_memory_allocated(dev)),
              "library_scratch_peak_bytes": tv.memory_stats()[1],
              "device_used_bytes_after": int(total_b - free_b), "device_total_bytes": int(total_b)}
    memory["peak_hbm_bytes"] = memory["torch_tensors_peak_bytes"] + memory["library_scratch_peak_bytes"]
    lib.tvgb_profile_read(buf, len(buf))
    lib.tvgb_profile_enable(0)
    prof = parse_profile(buf.value.decode())
    clocks = clk.summary()
    t_local = float(np.sum(times)) / 1e3
    t_max = t_local
    if dist:
        tt = torch.tensor([t_local], device=dev)
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        t_max = float(tt.item())
    value = (1 if strong else world) * args.steps * nvox / t_max

    # ---- end to end through the C ABI with pinned host buffers
    out_h = torch.empty((6,) + dims).pin_memory()
    ev_h = torch.empty(dims + (3,)).pin_memory()
    vec_h = torch.empty(dims + (3, 3)).pin_memory()
    vol_hn, out_hn, ev_hn, vec_hn = vol_h.numpy(), out_h.numpy(), ev_h.numpy(), vec_h.numpy()

    def step_e2e():
        if strong:
            slabs.pipeline3_slab(vol_hn, z0, z1, **skw)
        else:
            tv.pipeline3(vol_hn, outputs=(out_hn, ev_hn, vec_hn), **kw)

    step_e2e()
    if dist:
        dist.barrier()
    e2e_times = []
    for _ in range(args.steps):
        flush.zero_()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        step_e2e()
        e2e_times.append(time.perf_counter() - t0)
    t_e2e = float(np.sum(e2e_times))
    if dist:
        tt = torch.tensor([t_e2e], device=dev)
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        t_e2e = float(tt.item())
    e2e_value = (1 if strong else world) * args.steps * nvox / t_e2e
    h2d = vol_np.nbytes
    d2h = out_h.numel() * 4 + ev_h.numel() * 4 + vec_h.numel() * 4
    if strong:   # this rank's share: its input planes with halos, its output planes
        (il, ih), _ = slabs.halo_ranges(dims[0], z0, z1, cfg["sigma_st"], cfg["sigma"], 0.0, cfg["w"])
        h2d = vol_np[il:ih].nbytes
        d2h = d2h * (z1 - z0) // dims[0]

    # ---- roofline of the dominant kernel
    props = torch.cuda.get_device_properties(dev)
    sms = props.multi_processor_count
    max_mhz = clocks.get("sm_max_mhz") or 2070.0
    pk = fp32_peak(tv, sms, max_mhz)
    nl, tot_ms = prof.get("k_vote3_fast", (0, 0.0))
    roofline = None
    if nl:
        avg_s = tot_ms / nl / 1e3
        per_pair = FLOPS_PER_PAIR + (FLOPS_PER_PAIR_BALL if (cfg["ball"] or cfg["atv"]) else 0)
        flops = pairs_count(dims, cfg["w"] // 2, (z0, z1) if strong else None) * per_pair
        achieved = flops / avg_s / 1e12
        roofline = {"bound": "fp32", "kernel": "k_vote3_fast", "achieved": achieved, "peak": pk["nominal"],
                    "unit": "TFLOP/s", "frac": achieved / pk["nominal"], "peak_source": pk["source"],
                    "peak_measured_fma_chains": pk["measured"], "frac_of_measured_fma_chains":
                        achieved / pk["measured"],
                    **profiled_traffic("k_vote3_fast", args.config),
                    "flops_per_launch": flops, "flops_per_pair": per_pair, "avg_launch_ms": avg_s * 1e3,
                    "share_of_step": (tot_ms / (np.sum(times))) if np.sum(times) else None}
    nl, tot_ms = prof.get("k_sep_xy", (0, 0.0))
    taps = separable_taps(cfg["sigma"], cfg["w"] // 2)
    if nl and taps and not strong:
        # per voxel and weight: the 65 x sums and 121 y sums, a multiply-add each
        flops = nvox * taps * (65 + 121) * 2
        achieved = flops * args.steps / (tot_ms / 1e3) / 1e12
        roofline = {"bound": "fp32", "kernel": "k_sep_xy", "achieved": achieved, "peak": pk["nominal"],
                    "unit": "TFLOP/s", "frac": achieved / pk["nominal"], "peak_source": pk["source"],
                    "peak_measured_fma_chains": pk["measured"], "frac_of_measured_fma_chains":
                        achieved / pk["measured"],
                    **profiled_traffic("k_sep_xy", "c2", nvox),
                    "flops_per_step": flops, "flops_per_voxel": taps * (65 + 121) * 2,
                    "ms_per_step": tot_ms / args.steps, "launches_per_step": nl / args.steps,
                    "share_of_step": (tot_ms / (np.sum(times))) if np.sum(times) else None}

    # the structure tensor's kernel against the HBM roofline: 4 B in + 24 B out per voxel
    st_roof = None
    st_name = "k_st3_tma" if "k_st3_tma" in prof else "k_st3"
    nl_st, tot_st = prof.get(st_name, (0, 0.0))
    if nl_st:
        avg_st = tot_st / nl_st / 1e3
        hbm = measured_peaks()
        st_ach = nvox * 28 / avg_st / 1e9
        st_roof = {"bound": "hbm", "kernel": st_name, "achieved": st_ach, "peak": hbm["hbm_gbs"], "unit": "GB/s",
                   "frac": st_ach / hbm["hbm_gbs"], "peak_source": hbm["source"], "bytes_per_voxel": 28,
                   "avg_launch_ms": avg_st * 1e3}

    sur = None
    if rank == 0 and world == 1 and not args.no_surrogate and not strong and not cfg["atv"]:
        sur = surrogate_study(vol_d, cfg, args, dev)

    cpu = None
    accuracy = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        detail = {}
        t, nrec, th = cpu_reference_sample(vol_np, cfg, block=args.ref_block, seed=0, detail=detail)
        if not strong:
            # the same pipeline in precise mode (outside every timed region), for the FP64 comparison
            p_out = torch.empty_like(out_d)
            p_ev = torch.empty_like(ev_d)
            p_vec = torch.empty_like(vec_d)
            tv.pipeline3(vol_d, outputs=(p_out, p_ev, p_vec), parity=False, **kw)
            torch.cuda.synchronize()
            accuracy = accuracy_against_cpu(detail, cfg, out_d, ev_d, vec_d, th,
                                            precise=None if cfg["atv"] else (p_out, p_ev, p_vec))
            del p_out, p_ev, p_vec
        cpu = {"value": nrec / t, "unit": "voxels/s", "cores": th, "kind": "port",
               "sample": f"{args.ref_block}^3 interior receivers of the same volume (+ window halo), the reference's "
                         f"CPU algorithm ({'ATV, tensorvote.h:710' if cfg['atv'] else 'stick + ' + str(cfg['samples']) + '-sample plate'}"
                         f"{'; no ball: the reference has no TK ball' if cfg['ball'] else ''}) in oracle/, OpenMP over "
                         "receivers"}
    if rank == 0:
        line = {
            "metric": metric_for(cfg), "value": value, "unit": "voxels/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": 1e3 * t_max / args.steps, "higher_is_better": True,
            "scaling": "strong" if strong else "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": config_dict(cfg),
            "parallelism": (f"z-slabs x{world} (halo planes, no collective)" if strong else f"replicas x{world}"),
            "e2e": {"value": e2e_value, "unit": "voxels/s", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h},
            "gpu_launches": int(launches), "roofline": roofline, "cpu_baseline": cpu, "clocks": clocks,
            "kernels": {k: {"launches": v[0], "total_ms": v[1]} for k, v in prof.items()},
            "memory": memory, "surrogate": sur, "accuracy": accuracy,
            "structure_tensor_roofline": st_roof,
        }
        if world == 1 and not args.no_secondary and not strong:
            line["secondary"] = secondary_configs(args, local_rank)
        print(json.dumps(line), flush=True)
    if dist:
        dist.barrier()
        dist.destroy_process_group()


def secondary_configs(args, local_rank):
    """Compact measurements of the other workloads, after the headline's: C1
    (the 2D path, 512^2: value, e2e, FP32 roofline of the vote, errors
    against the reference's CPU algorithm) and C3 (2^27
    tensors in precise mode: value, HBM roofline of the eigensolver; no host
    round trip).  A few seconds of GPU time."""
    out = {}
    a1 = argparse.Namespace(**vars(args))
    # C1's CPU leg is a 192^2 crop (about a second): it gives the config's errors against the reference's algorithm
    a1.config, a1.size, a1.steps, a1.warmup = "c1", 0, 5, 3
    l1 = run_c1(a1, 0, 1, local_rank, emit=False)
    out["c1"] = {"workload": l1["config"]["workload"], "metric": l1["metric"], "value": l1["value"],
                 "unit": l1["unit"], "ms_per_step": l1["ms_per_step"], "e2e": l1["e2e"], "roofline": l1["roofline"],
                 "accuracy": l1["accuracy"], "cpu_baseline": l1["cpu_baseline"], "clocks": l1["clocks"]}
    a3 = argparse.Namespace(**vars(args))
    a3.config, a3.size, a3.steps, a3.warmup, a3.no_cpu_baseline = "c3", 0, 3, 3, True
    l3 = run_c3(a3, 0, 1, local_rank, emit=False, light=True)
    out["c3"] = {"workload": l3["config"]["workload"], "metric": l3["metric"], "value": l3["value"],
                 "unit": l3["unit"], "ms_per_step": l3["ms_per_step"], "roofline": l3["roofline"],
                 "fp64_refined_fraction": l3["fp64_refined_fraction"], "clocks": l3["clocks"]}
    return out


# ----------------------------------------------------------------------------- surrogate vs plain

def surrogate_study(vol_d, cfg, args, dev):
    """The learned plate vote against the plain 64-orientation integral and
    the exact closed form, in the same kernel skeleton, on a bounded interior
    block of the benchmark's own field (the structure tensor of the whole
    volume, cropped): stick exact in every mode, plate by the rule named.
    The network (28 features -> 64 -> 64 -> 64 -> 6, BF16 on tcgen05) is trained first,
    on the GPU, on 2^24 samples of the plain integral.  Errors are against
    the closed form, the exact integral (within 2e-6 of the FP64 oracle)."""
    import ctypes
    import torch
    import tiralib_gb300 as tv
    from tiralib_gb300 import surrogate as S
    lib = tv.lib()
    b = min(args.sur_block, cfg["n"])
    lo = (cfg["n"] - b) // 2
    F = tv.structure_tensor3(vol_d, cfg["sigma_st"], mode="same", layout="mat3")
    F = F[lo:lo + b, lo:lo + b, lo:lo + b].contiguous()
    t0 = time.perf_counter()
    X, T = S.samples(1 << 24, seed=4, device=dev)
    p = S.init_params(0)
    hist = S.train(p, X, T, batch=8192, steps=args.sur_steps, lr=args.sur_lr)
    torch.cuda.synchronize()
    t_train = time.perf_counter() - t0
    del X, T
    Xh, Th = S.samples(1 << 16, seed=77)
    Yh = S.evaluate(p, Xh)
    heldout = float(np.linalg.norm(Yh[:, :6] - Th[:, :6]) / np.linalg.norm(Th[:, :6]))
    buf = ctypes.create_string_buffer(1 << 14)
    kname = {"closed": "k_vote3_sur_closed", "plain64": "k_vote3_sur_plain64", "surrogate": "k_vote3_surtc"}
    runs = {"closed": ("closed", 1e-3), "plain64": ("plain64", 1e-3), "surrogate_judged": ("surrogate", 1e-3),
            "surrogate_judged_1e-2": ("surrogate", 1e-2), "surrogate_unjudged": ("surrogate", float("inf"))}
    if args.sur_modes:
        keep = set(args.sur_modes.split(",")) | {"closed"}      # the exact vote is the error reference
        runs = {k: v for k, v in runs.items() if k in keep}
    res, kms, stats = {}, {}, {}
    for key, (mode, tol) in runs.items():
        if args.sur_warm:
            S.vote3(F, cfg["sigma"], params=p, mode=mode, tol=tol, w=cfg["w"])      # warm-up
        lib.tvgb_profile_enable(1)
        lib.tvgb_profile_read(buf, len(buf))
        reps = args.sur_reps
        for _ in range(reps):
            o, _, _, st = S.vote3(F, cfg["sigma"], params=p, mode=mode, tol=tol, w=cfg["w"])
        torch.cuda.synchronize()
        lib.tvgb_profile_read(buf, len(buf))
        lib.tvgb_profile_enable(0)
        nl, ms = parse_profile(buf.value.decode()).get(kname[mode], (0, 0.0))
        kms[key] = ms / max(nl, 1)
        res[key] = o.cpu().numpy().reshape(-1, 9)[:, [0, 1, 2, 4, 5, 8]].astype(np.float64)
        stats[key] = st
    rates = (ctypes.c_double * 4)()
    lib.tvgb_pipe_rates(rates, None)
    ex = res["closed"]
    nex = np.linalg.norm(ex)
    err = {k: {"normwise": float(np.linalg.norm(v - ex) / nex), "max_abs_over_max": float(np.abs(v - ex).max() /
                                                                                         np.abs(ex).max())}
           for k, v in res.items() if k != "closed"}
    vps = {k: b ** 3 / (v / 1e3) for k, v in kms.items()}
    ratio = (lambda a, c: vps[a] / vps[c] if a in vps and c in vps else None)
    judged = stats.get("surrogate_judged")
    return {
        "sample": f"{b}^3 interior block of this field (structure tensor of the whole volume, cropped), sigma "
                  f"{cfg['sigma']:g}, w {cfg['w']}; stick exact, plate by the rule named; ball off",
        "network": f"28-64-64-64-6 GELU (inputs: direction, normal, flag and their degree-2 monomials), BF16 "
                   f"weights and activations, FP32 accumulation, tcgen05.mma with the "
                   f"activations in tensor memory; trained here on 2^24 plain-integral samples, {args.sur_steps} "
                   f"Adam steps of 8192 (lr {args.sur_lr:g}, cosine decay)",
        "train_s": t_train, "final_loss": float(np.mean(hist[-100:])), "heldout_rel_err": heldout,
        "kernel_ms": kms, "voxels_per_s": vps,
        "surrogate_vs_plain64": ratio("surrogate_unjudged", "plain64"),
        "surrogate_judged_vs_plain64": ratio("surrogate_judged", "plain64"),
        "closed_vs_plain64": ratio("closed", "plain64"),
        "rel_err_vs_exact": err,
        "judge": {"tol": 1e-3, "rule": "per CTA: the plate of its first 32 receivers against the exact plate, "
                                       "normwise over the 32, relative to their voted tensors",
                  "ctas": int(judged[0]) if judged else None,
                  "recomputed_exactly": int(judged[1]) if judged else None,
                  "recomputed_exactly_at_tol_1e-2": (int(stats["surrogate_judged_1e-2"][1])
                                                     if "surrogate_judged_1e-2" in stats else None)},
        "pipe_rates_per_sm_clock": {"fp32_fma": rates[0], "tanh_f32": rates[1], "tanh_bf16x2_results": rates[2],
                                    "sm_mhz": rates[3]},
    }


# ----------------------------------------------------------------------------- C3: batched 3x3 eigen

C3_METRIC = "batched 3x3 symmetric eigendecomposition tensors/s (FP32 + FP64 refinement of near-degenerate pairs)"


def eigen_batch_gpu(n, seed, dev, chunk=1 << 24):
    """n float32 tensors Q diag(l) Q^T on the GPU: Q a Haar rotation (random
    unit quaternion), l log-uniform in [1e-6, 1e3]; 10 % with a pair within
    1e-6 relative, 1 % fully degenerate (the C3 recipe)."""
    import torch
    out = torch.empty((n, 9), device=dev)
    g = torch.Generator(device=dev).manual_seed(seed)
    for s in range(0, n, chunk):
        m = min(chunk, n - s)
        q = torch.randn((m, 4), device=dev, generator=g, dtype=torch.float64)
        q = q / q.norm(dim=1, keepdim=True)
        w, x, y, z = q.unbind(1)
        Q = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                         2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                         2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], dim=1).view(m, 3, 3)
        lam = 10.0 ** (torch.rand((m, 3), device=dev, generator=g, dtype=torch.float64) * 9.0 - 6.0)
        k = torch.rand(m, device=dev, generator=g, dtype=torch.float64)
        pair = k < 0.10
        lam[pair, 1] = lam[pair, 0] * (1 + (torch.rand(int(pair.sum()), device=dev, generator=g,
                                                       dtype=torch.float64) * 2 - 1) * 1e-6)
        full = k >= 0.99
        lam[full, 1] = lam[full, 0]
        lam[full, 2] = lam[full, 0]
        M = (Q * lam[:, None, :]) @ Q.transpose(1, 2)
        out[s:s + m] = M.reshape(m, 9).float()
    return out


def eigen_errors(m9, ev, vec):
    """Errors against the FP64 oracle (Jacobi on the float32 input):
    eigenvalues normwise (|dl| / max|l|); eigenvector angle, separately for
    eigenvalues whose nearest neighbour is > 1e-3 |l_max| away and for those
    within (1e-9, 1e-3] |l_max| (near-degenerate pairs; the float32 input
    still determines them); and the backward error ||A V - V L|| / ||A||."""
    from oracle import oracle as O
    u = [0, 1, 2, 4, 5, 8]
    ref_ev, ref_vec = O.eig3_f64(m9[:, u].astype(np.float64))
    scale = np.abs(ref_ev).max(axis=1, keepdims=True)
    ev_err = (np.abs(ev - ref_ev) / scale).ravel()
    gaps = np.diff(ref_ev, axis=1) / scale
    gmin = np.full(ref_ev.shape, np.inf)           # relative gap to the nearest neighbour
    gmin[:, :2] = np.minimum(gmin[:, :2], gaps)
    gmin[:, 1:] = np.minimum(gmin[:, 1:], gaps)
    sep = gmin > 1e-3
    near = (gmin > 1e-9) & ~sep
    v64 = vec.astype(np.float64)
    v64 = v64 / np.linalg.norm(v64, axis=2, keepdims=True)
    dot = np.abs(np.einsum("nij,nij->ni", v64, ref_vec))
    crs = np.linalg.norm(np.cross(v64, ref_vec), axis=2)
    ang_all = np.arctan2(crs, dot)   # well conditioned at small angles, unlike arccos
    ang, ang_near = ang_all[sep], ang_all[near]
    A = m9.reshape(-1, 3, 3).astype(np.float64)
    V = vec.astype(np.float64)
    res = np.einsum("nij,nkj->nki", A, V) - ev.astype(np.float64)[:, :, None] * V
    bw = np.linalg.norm(res.reshape(len(A), -1), axis=1) / np.linalg.norm(A.reshape(len(A), -1), axis=1)
    stat = lambda x: {"max": float(np.max(x)), "median": float(np.median(x))} if len(x) else None
    return {"eigenvalue_normwise": stat(ev_err), "eigenvector_angle_rad": stat(ang),
            "eigenvector_angle_near_degenerate_rad": stat(ang_near), "n_near_degenerate": int(near.sum()),
            "backward": stat(bw), "n": int(len(m9))}


def run_c3(args, rank, world, local_rank, emit=True, light=False):
    import torch
    import tiralib_gb300 as tv
    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    n = 1 << args.size if args.size else 1 << 27
    mats = eigen_batch_gpu(n, 3 + rank, dev)
    ev = torch.empty((n, 3), device=dev)
    vec = torch.empty((n, 3, 3), device=dev)
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)
    lib = tv.lib()
    buf = ctypes.create_string_buffer(1 << 14)

    def timed(precise):
        for _ in range(args.warmup):
            tv.api.call("tvgb_eig3", tv.api._ptr(mats), 9, n, tv.api._ptr(ev), tv.api._ptr(vec), 1, int(precise),
                        None, tv.api._stream_for(mats))
        torch.cuda.synchronize()
        lib.tvgb_profile_enable(1)
        lib.tvgb_profile_read(buf, len(buf))
        ts = []
        l0 = tv.launch_count()
        for _ in range(args.steps):
            flush.zero_()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            tv.api.call("tvgb_eig3", tv.api._ptr(mats), 9, n, tv.api._ptr(ev), tv.api._ptr(vec), 1, int(precise),
                        None, tv.api._stream_for(mats))
            e1.record()
            e1.synchronize()
            ts.append(e0.elapsed_time(e1))
        launches = tv.launch_count() - l0
        lib.tvgb_profile_read(buf, len(buf))
        lib.tvgb_profile_enable(0)
        return float(np.sum(ts)) / 1e3, launches, parse_profile(buf.value.decode())

    # precision on a 2^16 sample of the timed runs' own outputs (every chunk of the batch)
    idx = torch.randperm(n, device=dev, generator=torch.Generator(device=dev).manual_seed(9))[: 1 << 16]
    with ClockSampler(gpu_index_for(local_rank)) as clk:
        t_precise, launches, prof = timed(True)
    clocks = clk.summary()
    _, _, nref = tv.eig3(mats[: 1 << 20], precise=True)
    t_parity, err_precise, err_parity, e2e = None, None, None, None
    if not light:
        ev_p, vec_p = ev[idx].cpu().numpy(), vec[idx].cpu().numpy()
        t_parity, _, prof_par = timed(False)
        ev_r, vec_r = ev[idx].cpu().numpy(), vec[idx].cpu().numpy()
        m_h = mats[idx].cpu().numpy()
        err_precise = eigen_errors(m_h, ev_p, vec_p)
        err_parity = eigen_errors(m_h, ev_r, vec_r)
        # end to end with pinned host buffers
        mats_h = mats.cpu().pin_memory()
        ev_h = torch.empty((n, 3)).pin_memory()
        vec_h = torch.empty((n, 3, 3)).pin_memory()
        mn, evn, vecn = mats_h.numpy(), ev_h.numpy(), vec_h.numpy()
        # one full-size untimed call: the library's memory pool grows to the chunk ring's size once
        tv.api.call("tvgb_eig3", tv.api._ptr(mn), 9, n, tv.api._ptr(evn), tv.api._ptr(vecn), 1, 1, None, None)
        e2e = []
        for _ in range(max(1, min(args.steps, 3))):
            t0 = time.perf_counter()
            tv.api.call("tvgb_eig3", tv.api._ptr(mn), 9, n, tv.api._ptr(evn), tv.api._ptr(vecn), 1, 1, None, None)
            e2e.append(time.perf_counter() - t0)
    peaks = measured_peaks()
    # the precise call is one k_eig3 launch (FP32 solve, FP64 refinement of the flagged tensors from the tile
    # in shared memory): its roofline is the call's algorithmic bytes over the kernel's time per call
    nl, tot = prof.get("k_eig3", (0, 0.0))
    bytes_per = 36 + 12 + 36
    roof = None
    if nl:
        avg = tot / args.steps / 1e3
        ach = n * bytes_per / avg / 1e9
        roof = {"bound": "hbm", "kernel": "k_eig3 (precise, per call)", "achieved": ach,
                "peak": peaks["hbm_gbs"], "unit": "GB/s", "frac": ach / peaks["hbm_gbs"],
                "peak_source": peaks["source"], "bytes_per_tensor": bytes_per, "avg_call_kernel_ms": avg * 1e3}
        roof.update(profiled_traffic("k_eig3", "c3", n))
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        v, th, desc = cpu_eigen_sample()
        cpu = {"value": v, "unit": "tensors/s", "cores": th, "kind": "port", "sample": desc}
    line = None
    if rank == 0:
        line = {
            "metric": C3_METRIC, "value": world * args.steps * n / t_precise, "unit": "tensors/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * t_precise / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32 (f64 refinement)",
            "data": "synthetic",
            "config": {"workload": f"C3: 2^{int(np.log2(n))} tensors Q diag(l) Q^T, Haar Q, l log-uniform [1e-6, 1e3],"
                                   " 10% near-degenerate pair, 1% fully degenerate; mat3 in, eigenvalues + "
                                   "cartesian eigenvectors out", "tensors": n,
                       "l2_flush": "256 MiB write between timed steps (outside the events)"},
            "parity_mode_tensors_per_s": args.steps * n / t_parity if t_parity else None,
            "fp64_refined_fraction": nref / float(1 << 20),
            "errors_vs_fp64": {"precise": err_precise, "parity": err_parity},
            "e2e": ({"value": n / float(np.mean(e2e)), "unit": "tensors/s", "h2d_bytes_per_step": n * 36,
                     "d2h_bytes_per_step": n * 48} if e2e else None),
            "gpu_launches": int(launches), "roofline": roof, "cpu_baseline": cpu, "clocks": clocks,
            "kernels": {k: {"launches": v[0], "total_ms": v[1]} for k, v in prof.items()},
        }
        if emit:
            print(json.dumps(line), flush=True)
    del mats, ev, vec
    torch.cuda.empty_cache()
    return line


def cpu_eigen_sample(n=1 << 20):
    from oracle import oracle as O
    from tiralib_gb300 import workloads as W
    m9 = W.eigen_batch(n, seed=4)
    th = os.cpu_count() or 1
    O.eig3_threads(m9[:4096], th)
    t0 = time.perf_counter()
    O.eig3_threads(m9, th)
    t = time.perf_counter() - t0
    return n / t, th, (f"2^{int(np.log2(n))} C3-recipe tensors through eigen.h's CPU solve (evals3_symmetric + "
                       f"evec3_symmetric, C port), OpenMP over tensors")


def measured_peaks():
    path = os.path.join(HERE, "MEASURED_PEAKS.json")
    try:
        d = json.load(open(path))
        return {"hbm_gbs": float(d["hbm_gbs"]), "source": "measured (MEASURED_PEAKS.json hbm_gbs, copy)"}
    except Exception:
        return {"hbm_gbs": 6800.0, "source": "fallback 6.8 TB/s"}


def run_c3_reference(args, rank):
    if rank != 0:
        return
    vals = []
    th, desc = 1, ""
    for _ in range(args.warmup):
        cpu_eigen_sample()
    for _ in range(args.steps):
        v, th, desc = cpu_eigen_sample()
        vals.append(v)
    value = float(np.mean(vals))
    print(json.dumps({"impl": "reference", "metric": C3_METRIC, "value": value, "unit": "tensors/s",
                      "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
                      "ms_per_step": 1e3 * (1 << 20) / value, "higher_is_better": True, "scaling": "weak",
                      "vs_baseline": None, "dtype": "f32", "data": "synthetic",
                      "config": {"workload": "C3 eigen, bounded sample"},
                      "cpu_baseline": {"value": value, "unit": "tensors/s", "cores": th, "kind": "port",
                                       "sample": desc},
                      "e2e": {"value": value, "unit": "tensors/s", "h2d_bytes_per_step": 0,
                              "d2h_bytes_per_step": 0}}), flush=True)


# ----------------------------------------------------------------------------- C1: 2D

C1_METRIC = "2D tensor-vote pixels/s (structure tensor sigma 1 -> stick+plate vote sigma 3 -> 2x2 eigen)"


def run_c1(args, rank, world, local_rank, emit=True):
    import torch
    import tiralib_gb300 as tv
    from tiralib_gb300 import workloads as W
    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    size = args.size or 512
    img_np = W.curve_image(size, seed=1 + rank)
    img = torch.from_numpy(img_np).to(dev)
    n = img_np.size
    st = torch.empty((size, size, 4), device=dev)
    voted = torch.empty((size, size, 4), device=dev)
    ev = torch.empty((n, 2), device=dev)
    th = torch.empty((n, 2), device=dev)
    sigma, w, samples = 3.0, 19, 20
    S = ctypes.c_void_p
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)

    def step(src, st_, vo, e, t, stream):
        d = (ctypes.c_uint * 2)()
        tv.api.call("tvgb_structure_tensor2", tv.api._ptr(src), size, size, 1.0, 1, tv.api._ptr(st_), d, stream)
        tv.api.call("tvgb_tensorvote", tv.api._ptr(vo), tv.api._ptr(st_), sigma, 0.0, 1, w, size, size, 1, 1,
                    samples, 0, stream)
        tv.api.call("tvgb_evals2_symmetric", tv.api._ptr(vo), n, tv.api._ptr(e), stream)
        tv.api.call("tvgb_evecs2polar_symmetric", tv.api._ptr(vo), tv.api._ptr(e), n, tv.api._ptr(t), stream)

    stream = S(torch.cuda.current_stream().cuda_stream)
    for _ in range(args.warmup):
        step(img, st, voted, ev, th, stream)
    torch.cuda.synchronize()
    lib = tv.lib()
    buf = ctypes.create_string_buffer(1 << 14)
    # per-kernel durations (CUDA events inside the library) from calls made one by one
    lib.tvgb_profile_enable(1)
    lib.tvgb_profile_read(buf, len(buf))
    ts_calls = []
    for _ in range(args.steps):
        flush.zero_()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        step(img, st, voted, ev, th, stream)
        e1.record()
        e1.synchronize()
        ts_calls.append(e0.elapsed_time(e1))
    lib.tvgb_profile_read(buf, len(buf))
    lib.tvgb_profile_enable(0)
    prof = parse_profile(buf.value.decode())
    # the timed step: the same four library calls captured once as a CUDA graph and replayed, so the
    # ~8 short kernels of a 512^2 step run back to back without host work between their launches
    graph = torch.cuda.CUDAGraph()
    l_cap = tv.launch_count()
    with torch.cuda.graph(graph):
        step(img, st, voted, ev, th, S(torch.cuda.current_stream().cuda_stream))
    kernels_per_step = tv.launch_count() - l_cap
    for _ in range(args.warmup):
        graph.replay()
    torch.cuda.synchronize()
    ts = []
    with ClockSampler(gpu_index_for(local_rank)) as clk:
        for _ in range(args.steps):
            flush.zero_()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            graph.replay()
            e1.record()
            e1.synchronize()
            ts.append(e0.elapsed_time(e1))
    launches = kernels_per_step * args.steps
    free_b, total_b = torch.cuda.mem_get_info(dev)
    memory = {"torch_tensors_peak_bytes": int(torch.cuda.max_memory_allocated(dev)),
              "library_scratch_peak_bytes": tv.memory_stats()[1],
              "device_used_bytes_after": int(total_b - free_b), "device_total_bytes": int(total_b)}
    memory["peak_hbm_bytes"] = memory["torch_tensors_peak_bytes"] + memory["library_scratch_peak_bytes"]
    t = float(np.sum(ts)) / 1e3
    # end to end: host image in, host voted field + eigenpairs out
    img_h = torch.from_numpy(img_np).pin_memory().numpy()
    st_h = torch.empty((size, size, 4)).pin_memory().numpy()
    vo_h = torch.empty((size, size, 4)).pin_memory().numpy()
    ev_h = torch.empty((n, 2)).pin_memory().numpy()
    th_h = torch.empty((n, 2)).pin_memory().numpy()
    step(img_h, st_h, vo_h, ev_h, th_h, None)
    e2e = []
    for _ in range(args.steps):
        t0 = time.perf_counter()
        step(img_h, st_h, vo_h, ev_h, th_h, None)
        e2e.append(time.perf_counter() - t0)
    # 2D pair as k_vote2_tks computes it (FMA = 2): stick q.d 3, q^2 1, D = c1 + (c2 - c1) q^2 2,
    # -2 q.d 1, R q = q - 2 (q.d) d 4, f 1, f Rq 2, 3 accumulations 6; plate 3 FMAs 6: 26 flops
    # (the reference's literal expressions, with the entry's (Ra, Rb, Rc) product, take 30)
    pairs = 1
    for d in (size, size):
        pairs *= sum(min(d - 1, x + w // 2) - max(0, x - w // 2) + 1 for x in range(d))
    nl, tot = prof.get("k_vote2_tk", (0, 0.0))
    roof = None
    if nl:
        avg = tot / nl / 1e3
        props = torch.cuda.get_device_properties(dev)
        pk = fp32_peak(tv, props.multi_processor_count, 2070.0)
        ach = pairs * 26 / avg / 1e12
        roof = {"bound": "fp32", "kernel": "k_vote2_tk", "achieved": ach, "peak": pk["nominal"], "unit": "TFLOP/s",
                "frac": ach / pk["nominal"], "peak_measured_fma_chains": pk["measured"],
                "frac_of_measured_fma_chains": ach / pk["measured"],
                "flops_per_pair": 26, "avg_launch_ms": avg * 1e3, "peak_source": pk["source"],
                **profiled_traffic("k_vote2_tk", "c1")}
    cpu = accuracy = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        from oracle import oracle as O
        cs = min(192, size)                                  # crop edge
        crop = img_np[:cs, :cs]
        t0 = time.perf_counter()
        st_c = O.structure_tensor2(crop, 1.0, 1)
        vo_c = O.tensorvote2(st_c, sigma, 0.0, 1, w, samples=samples)
        e_c = O.evals2(vo_c)
        th_c = O.evecs2polar(vo_c, e_c)
        tc = time.perf_counter() - t0
        cpu = {"value": crop.size / tc, "unit": "pixels/s", "cores": 1, "kind": "port",
               "sample": f"{cs}x{cs} crop: the reference's CPU 2D path (tira::cpu::tensorvote's algorithm, single "
                         "thread as shipped) incl. structure tensor and eigenpairs"}
        # the crop's interior (its window and blur halo away from the crop's edges) sees the same pixels as
        # the full image: the GPU's end-to-end outputs there against the reference's CPU algorithm
        m = w // 2 + 4
    if cpu is not None and cs > 2 * m:
        g_vo = vo_h[m:cs - m, m:cs - m].reshape(-1, 4).astype(np.float64)
        r_vo = np.asarray(vo_c)[m:cs - m, m:cs - m].reshape(-1, 4).astype(np.float64)
        pix = (np.arange(m, cs - m)[:, None] * size + np.arange(m, cs - m)[None, :]).ravel()
        g_ev, r_ev = ev_h[pix].astype(np.float64), np.asarray(e_c).reshape(-1, 2)[
            (np.arange(m, cs - m)[:, None] * cs + np.arange(m, cs - m)[None, :]).ravel()].astype(np.float64)
        g_th = th_h[pix].astype(np.float64)
        r_th = np.asarray(th_c).reshape(-1, 2)[
            (np.arange(m, cs - m)[:, None] * cs + np.arange(m, cs - m)[None, :]).ravel()].astype(np.float64)
        vr = np.linalg.norm(g_vo - r_vo, axis=1) / np.maximum(np.linalg.norm(r_vo, axis=1), 1e-30)
        er = np.abs(g_ev - r_ev).max(axis=1) / np.maximum(np.abs(r_ev).max(axis=1), 1e-30)
        da = np.abs(g_th - r_th) % np.pi                   # eigenvector angles, up to sign
        da = np.minimum(da, np.pi - da).max(axis=1)
        accuracy = {"pixels": int(len(pix)), "voted_vs_reference_cpu": {"per_pixel_max": float(vr.max()),
                                                                       "per_pixel_median": float(np.median(vr))},
                    "eigenvalues_vs_reference_cpu": {"max": float(er.max()), "median": float(np.median(er))},
                    "eigenvector_angle_rad_vs_reference_cpu": {"max": float(da.max()), "median": float(np.median(da))}}
    line = None
    if rank == 0:
        line = {
            "metric": C1_METRIC, "value": world * args.steps * n / t, "unit": "pixels/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * t / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": f"C1: {size}^2 image of 32 random cubic Bezier curves (width 1.5) + N(0, 0.05); "
                                   "np.gradient structure tensor, Gaussian sigma 1 (same size); TK stick + plate "
                                   "vote sigma 3, w 19, samples 20; 2x2 eigenpairs", "pixels": n,
                       "step": "the four library calls captured once as a CUDA graph, replayed per step",
                       "l2_flush": "256 MiB write between timed steps (outside the events)"},
            "ms_per_step_calls_one_by_one": float(np.mean(ts_calls)),
            "e2e": {"value": n / float(np.mean(e2e)), "unit": "pixels/s", "h2d_bytes_per_step": img_np.nbytes,
                    "d2h_bytes_per_step": st_h.nbytes + vo_h.nbytes + ev_h.nbytes + th_h.nbytes},
            "gpu_launches": int(launches), "roofline": roof, "cpu_baseline": cpu, "accuracy": accuracy,
            "clocks": clk.summary(),
            "kernels": {k: {"launches": v[0], "total_ms": v[1]} for k, v in prof.items()},
            "memory": memory,
        }
        if emit:
            print(json.dumps(line), flush=True)
    return line


def run_c1_reference(args, rank):
    """The reference's CPU 2D path (oracle port of tira::cpu::tensorvote,
    single thread as shipped) on the full C1 image, per step."""
    if rank != 0:
        return
    from oracle import oracle as O
    from tiralib_gb300 import workloads as W
    size = args.size or 512
    img = W.curve_image(size, seed=1)
    sigma, w, samples = 3.0, 19, 20

    def step():
        st = O.structure_tensor2(img, 1.0, 1)
        vo = O.tensorvote2(st, sigma, 0.0, 1, w, samples=samples)
        e = O.evals2(vo)
        O.evecs2polar(vo, e)

    for _ in range(args.warmup):
        step()
    ts = []
    for _ in range(args.steps):
        t0 = time.perf_counter()
        step()
        ts.append(time.perf_counter() - t0)
    value = args.steps * img.size / float(np.sum(ts))
    print(json.dumps({
        "impl": "reference", "metric": C1_METRIC, "value": value, "unit": "pixels/s", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * float(np.mean(ts)),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": f"C1: {size}^2 curve image, TK stick + plate vote sigma 3, w 19, samples 20, 2x2 "
                               "eigenpairs", "pixels": img.size},
        "cpu_baseline": {"value": value, "unit": "pixels/s", "cores": 1, "kind": "port",
                         "sample": f"the full {size}^2 image per step: structure tensor, tira::cpu::tensorvote's "
                                   "algorithm, eigenpairs (single thread, as shipped)"},
        "e2e": {"value": value, "unit": "pixels/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }), flush=True)


def main():
    ap = argparse.ArgumentParser(description=__doc__, formatter_class=argparse.RawDescriptionHelpFormatter)
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--ref-block", type=int, default=12, help="edge of the CPU reference's receiver block")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-surrogate", action="store_true", help="skip the surrogate-vs-plain study")
    ap.add_argument("--no-secondary", action="store_true", help="skip the C1 / C3 measurements after the headline")
    ap.add_argument("--sur-block", type=int, default=128, help="edge of the surrogate study's interior block")
    ap.add_argument("--sur-reps", type=int, default=1, help="timed launches per mode of the surrogate study")
    ap.add_argument("--sur-warm", type=int, default=1, help="1: one untimed launch per mode first")
    ap.add_argument("--sur-modes", default="", help="comma-separated subset of the surrogate study's modes "
                                                    "(plain64, surrogate_judged, surrogate_judged_1e-2, "
                                                    "surrogate_unjudged); the exact vote always runs")
    ap.add_argument("--sur-steps", type=int, default=300000, help="Adam steps of the surrogate's training")
    ap.add_argument("--sur-lr", type=float, default=3e-3, help="peak learning rate of the surrogate's training")
    ap.add_argument("--config", choices=["c2", "c4", "c5", "c3", "c1"], default="c4",
                    help="c4: 3D pipeline at 384^3, sigma 4, the surrogate study's field (the headline); c2: the same "
                         "at 256^3; c5: 512^3 tubes + sheets, sigma 6, stick + plate + ball (capacity); c3: batched "
                         "3x3 eigen; c1: 2D pipeline")
    ap.add_argument("--atv", action="store_true", help="c2/c4/c5: vote with ATV (analytical tensor voting, "
                                                       "tensorvote.h:710) instead of TK")
    ap.add_argument("--split", choices=["replicas", "slabs"], default="replicas",
                    help="N > 1: independent replicas (weak scaling) or z-slabs of one volume (strong scaling)")
    ap.add_argument("--size", type=int, default=0, help="c2/c4/c5: volume edge (default 256/384/512); c3: log2 of "
                                                        "the tensor count (default 27); c1: image edge (default "
                                                        "512). Smaller sizes are for profiler captures")
    args = ap.parse_args()
    if args.warmup < 3:
        ap.error("--warmup must be >= 3")
    rank, world, local_rank = dist_env()
    if args.config == "c3":
        return run_c3_reference(args, rank) if args.impl == "reference" else run_c3(args, rank, world, local_rank)
    if args.config == "c1":
        return run_c1_reference(args, rank) if args.impl == "reference" else run_c1(args, rank, world, local_rank)
    if args.impl == "reference":
        run_reference(args, rank)
        return
    run_ours(args, rank, world, local_rank)


if __name__ == "__main__":
    main()
