#!/usr/bin/env python3
"""Benchmark of the two-electron hot path: direct RHF on a seeded (H2O)16 cluster.

Workload (the reference metric's single-GPU configuration): 16 water monomers on a
4x4x1 lattice at 3.0 Angstrom, rigidly rotated (uniform quaternions) and jittered
(+-0.3 Angstrom), seed 16; basis 6-31G** with Cartesian d (400 functions, 192
shells); direct SCF with Schwarz x density screening at 1e-12 (formPT semantics,
incremental Fock builds); FP64.  Synthetic data: the geometry is generated, no
dataset is involved.

One *step* is one RHF iteration with a Fock build (G(P - P_old) on the GPU,
symmetrised incremental update, DIIS, eigensolve, density, energy).  W warm-up
iterations run on a first SCF; the K timed steps are iterations 1..K of a fresh SCF
from the core guess (iteration 0 only diagonalises the core Hamiltonian).
Between timed steps a 512 MB buffer is written to flush the 129 MB L2.

Printed (rank 0, one JSON line):
  value      Fock builds/s (= RHF iterations/s), device-timed with CUDA events
  e2e        the same metric through the reference-facing API formPT(P, P_old,
             bfs, nbasis, screen, tol) with host arrays in and out
  time_to_converge_s  Molecule(geometry, basis).RHF(direct=True) wall time (conver 1e-8)
  roofline   FP64-pipe roofline of the dominant class kernel (live CUDA events; the
             FP64 FLOPs the kernels issue, counted from the code's structure and the
             build's counters by mmd/flop_model.py, with the algorithm's useful FLOPs
             and the dense reference model beside them, per class; peak measured
             live by mmdg_measure_peaks)
  cpu_baseline  the reference's Cython formPT (oracle/_ref) on the host cores, a
             bounded sample extrapolated to this workload (see cpu_sample())

``--impl reference`` times the reference's CPU implementation alone (rank 0).
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import tempfile
import threading
import time

REPO = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(REPO, "mcmurchie-davidson_gb300")
ORACLE = os.path.join(REPO, "oracle")

WORKLOAD = {"workload": "(H2O)16 6-31G** direct RHF", "n_water": 16, "lattice": "4x4x1", "spacing_A": 3.0,
            "jitter_A": 0.3, "seed": 16, "basis": "6-31G**", "nbasis": 400, "schwarz": 1e-12}
# Average number of function quartets that pass the reference's screening per Fock
# build over iterations 1..20 of the workload above (the GPU arm counts them with
# the same rule and prints its own figure as config.fq_per_build).  Used by the
# reference arm, which cannot run the 400-function SCF itself.
FQ_PER_BUILD = 198282802.0
# DRAM bytes (read + write) per launch of the two largest class kernels on this workload:
# launch 5 of each (an early Fock build of the warm-up SCF) in one ncu capture
# (dram__bytes_read.sum + dram__bytes_write.sum; summary and command in
# profiles/k_fock_1000_full_h2o16.md).
DRAM_BYTES_PER_LAUNCH = {"1000": 50.10e6, "1110": 16.26e6}
# FP64-pipe busy fraction of the same launch over its elapsed cycles
# (sm__pipe_fp64_cycles_active.avg.pct_of_peak_sustained_elapsed, same capture)
FP64_PIPE_BUSY = {"1000": 0.819, "1110": 0.652}


def _env():
    return int(os.environ.get("RANK", 0)), int(os.environ.get("WORLD_SIZE", 1)), int(os.environ.get("LOCAL_RANK", 0))


# ------------------------------------------------------------------------------ ranks
def max_over_ranks(t_local: float, device: str = "cpu") -> float:
    """The slowest rank's time (all-reduce MAX); the local time without a process group."""
    import torch
    import torch.distributed as dist
    if not (dist.is_available() and dist.is_initialized()) or dist.get_world_size() == 1:
        return float(t_local)
    t = torch.tensor([float(t_local)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def replica_throughput(world: int, units_per_rank: int, t_max: float) -> float:
    """Whole-job throughput of independent replicas: all ranks' units over the slowest
    rank's time (weak scaling: every rank runs the full workload)."""
    return world * units_per_rank / t_max


# ------------------------------------------------------------------------------ clocks
class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.lines = []

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except FileNotFoundError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, mx, reasons = [], [], set()
        names = ["active", "hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            p = [x.strip() for x in ln.split(",")]
            if len(p) < 9:
                continue
            try:
                sm.append(float(p[1]))
                mx.append(float(p[2]))
            except ValueError:
                continue
            for n, v in zip(names[1:], p[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        sm.sort()
        return {"sm_mhz": sm[len(sm) // 2] if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(sm)}


# ------------------------------------------------------------------------------ CPU sample
def _ref_worker_init(spec_path):
    global _W
    with open(spec_path) as f:
        spec = json.load(f)
    import numpy as np
    kind = spec["kind"]
    if kind == "reference":
        sys.path.insert(0, os.path.join(ORACLE, "_ref"))
        from mmd.integrals.twoe import Basis
        from mmd.integrals.fock import formPT
        bfs = [Basis(np.array(o), np.array(s), len(e), np.array(e), np.array(c)) for o, s, e, c in spec["bfs"]]
        screen = {i: v for i, v in enumerate(spec["screen"])}
    else:
        sys.path.insert(0, ORACLE)
        import oracle as O
        bfs = [O.Basis(o, s, len(e), e, c) for o, s, e, c in spec["bfs"]]
        formPT = O.formPT
        screen = np.array(spec["screen"])
    P = np.array(spec["P"], dtype=complex)
    _W = (formPT, bfs, screen, P, len(bfs))


def _ref_worker_run(mode):
    import numpy as np
    formPT, bfs, screen, P, N = _W
    Pold = P if mode == "skip" else np.zeros_like(P)
    t0 = time.perf_counter()
    formPT(P, Pold, bfs, N, screen, 1e-12)
    return time.perf_counter() - t0


def cpu_sample(spec_path, cores, steps, warmup):
    """Time the reference formPT on water/6-31G** in `cores` processes.

    Two calls per process and step: dP = 0 (every candidate quartet is screened
    out: the per-candidate screening cost of formPT's Python loop) and dP = P1 (the
    reference's first-iteration density: nearly every quartet survives).  The
    per-build time of the target is then  n_cand * t_skip + n_surv * t_eri  with
    t_eri = (t_full - t_skip) / n_surv_monomer.  Prints one JSON object."""
    import multiprocessing as mp
    with open(spec_path) as f:
        spec = json.load(f)
    ctx = mp.get_context("spawn")
    with ctx.Pool(cores, initializer=_ref_worker_init, initargs=(spec_path,)) as pool:
        for _ in range(max(warmup, 1)):
            pool.map(_ref_worker_run, ["skip"] * cores)
        t_skip, t_full = [], []
        for _ in range(steps):
            t_skip.append(max(pool.map(_ref_worker_run, ["skip"] * cores)))
            t_full.append(max(pool.map(_ref_worker_run, ["full"] * cores)))
    ts, tf = sum(t_skip) / len(t_skip), sum(t_full) / len(t_full)
    n_cand_m, n_surv_m = spec["n_cand_monomer"], spec["n_surv_monomer"]
    t_cand = ts / n_cand_m
    t_eri = max(tf - ts, 1e-12) / n_surv_m
    t_build = spec["n_cand_target"] * t_cand + spec["n_surv_target"] * t_eri
    out = {"kind": spec["kind"], "cores": cores, "t_skip_s": ts, "t_full_s": tf, "t_candidate_s": t_cand,
           "t_eri_s": t_eri, "t_build_1core_s": t_build, "builds_per_s": cores / t_build,
           "quartets_per_s_1core": 1.0 / t_eri, "steps": steps}
    anchor = spec.get("anchor")
    if anchor:
        # one whole formPT call of (H2O)2 on one core against the extrapolation's
        # prediction for it (the same per-candidate and per-survivor costs)
        with ctx.Pool(1, initializer=_ref_worker_init, initargs=(anchor["spec_path"],)) as pool:
            t_anchor = pool.map(_ref_worker_run, ["full"])[0]
        pred = anchor["n_cand"] * t_cand + anchor["n_surv"] * t_eri
        out["anchor"] = {"workload": anchor["workload"], "candidates": anchor["n_cand"], "survivors": anchor["n_surv"],
                         "measured_s": t_anchor, "predicted_s": pred, "measured_over_predicted": t_anchor / pred}
    print(json.dumps(out))


def _monomer_spec(kind):
    """Basis (raw coefficients), Schwarz table and first-iteration density of water/6-31G**
    for the CPU sample; all from the repository (tests/golden holds the reference's own run)."""
    import numpy as np
    sys.path.insert(0, PKG)
    from mmd.molecule import Molecule
    g = np.load(os.path.join(REPO, "tests", "golden", "mol_water_631gss.npz"))
    m = Molecule(str(g["geometry"]), "6-31gss")
    bfs = []
    for atom in m.atoms:
        for momentum, prims in m.basis_data[atom.charge]:
            ex = [e for e, c in prims]
            co = [c for e, c in prims]
            for sh in m.momentum2shell(momentum):
                bfs.append((list(map(float, atom.origin)), list(sh), ex, co))
    N = len(bfs)
    P1 = g["formPT0_P"]
    scr = g["screen"]
    n_cand, n_surv = _formpt_counts(P1, scr)
    return {"kind": kind, "bfs": bfs, "screen": scr.tolist(), "P": P1.tolist(),
            "n_cand_monomer": n_cand, "n_surv_monomer": n_surv}


def _formpt_counts(P, scr, tol=1e-12):
    """Candidate and surviving function quartets of one formPT call with dP = P: the
    reference's screening rule (fock.pyx:46-57) over its canonical quartets."""
    import numpy as np
    N = P.shape[0]
    sq = np.sqrt(scr)
    iu = np.array([(i, j) for i in range(N) for j in range(i + 1)])
    d = np.abs(P)
    n_surv = 0
    for a in range(len(iu)):
        i, j = iu[a]
        kl = iu[: a + 1]
        k, l = kl[:, 0], kl[:, 1]
        dm = np.maximum.reduce([np.full(len(kl), 4 * d[i, j]), 4 * d[k, l], d[i, k], d[i, l], d[j, k], d[j, l]])
        n_surv += int(np.sum(sq[a] * sq[: a + 1] * dm >= tol))
    npair = N * (N + 1) // 2
    return npair * (npair + 1) // 2, n_surv


def _anchor_spec(kind):
    """The (H2O)2 / 6-31G** formPT call of tests/golden/h2o2_631gss_formpt.npz (the
    first call of the reference's own direct RHF) in the worker's format."""
    import numpy as np
    sys.path.insert(0, PKG)
    from mmd.molecule import Molecule
    g = np.load(os.path.join(REPO, "tests", "golden", "h2o2_631gss_formpt.npz"))
    m = Molecule(str(g["geometry"]), "6-31gss")
    bfs = []
    for atom in m.atoms:
        for momentum, prims in m.basis_data[atom.charge]:
            ex = [e for e, c in prims]
            co = [c for e, c in prims]
            for sh in m.momentum2shell(momentum):
                bfs.append((list(map(float, atom.origin)), list(sh), ex, co))
    n_cand, n_surv = _formpt_counts(g["P"], g["screen"])
    return {"kind": kind, "bfs": bfs, "screen": g["screen"].tolist(), "P": g["P"].tolist(),
            "n_cand": n_cand, "n_surv": n_surv, "workload": f"(H2O)2 6-31G** (N={len(bfs)}), one formPT call, one core"}


def run_cpu_sample(n_cand_target, n_surv_target, steps, warmup, cores=None):
    kind = "reference" if os.path.isdir(os.path.join(ORACLE, "_ref", "mmd", "integrals")) and any(
        f.startswith("fock") and f.endswith(".so") for f in os.listdir(os.path.join(ORACLE, "_ref", "mmd", "integrals"))
    ) else "port"
    if kind == "port":
        subprocess.check_call(["make", "-s", "-C", ORACLE, "liboracle.so"])
    spec = _monomer_spec(kind)
    spec["n_cand_target"] = n_cand_target
    spec["n_surv_target"] = n_surv_target
    cores = cores or os.cpu_count()
    aspec = _anchor_spec(kind)
    with tempfile.NamedTemporaryFile("w", suffix=".json", delete=False) as f:
        json.dump(aspec, f)
        apath = f.name
    spec["anchor"] = {"spec_path": apath, "n_cand": aspec["n_cand"], "n_surv": aspec["n_surv"],
                      "workload": aspec["workload"]}
    with tempfile.NamedTemporaryFile("w", suffix=".json", delete=False) as f:
        json.dump(spec, f)
        path = f.name
    try:
        out = subprocess.run([sys.executable, os.path.abspath(__file__), "--cpu-sample", path, "--cores", str(cores),
                              "--steps", str(steps), "--warmup", str(warmup)],
                             capture_output=True, text=True, check=True, env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
    finally:
        os.unlink(path)
        os.unlink(apath)
    res = json.loads(out.stdout.strip().splitlines()[-1])
    res["sample"] = (f"reference formPT on water/6-31G** (N=25, {spec['n_cand_monomer']} candidate and "
                     f"{spec['n_surv_monomer']} surviving quartets) in {cores} processes, dP=0 and dP=P1 per step; "
                     f"extrapolated to {n_cand_target:.4g} candidates and {n_surv_target:.4g} survivors per build")
    return res


# ------------------------------------------------------------------------------ batched (config 3)
def batched_bench(nmol=1024, reps=5, sample_per_molecule=128, seed=3, parity_sample=128):
    """1024 seeded (H2O)n clusters, n ~ U{1..8}, 6-31G: one batched, graph-replayed and
    autotuned Fock launch for all molecules vs per-molecule launches, and the batched
    RHF to convergence."""
    import numpy as np
    import torch
    from mmd import autotune
    from mmd.batch import BatchRHF, per_molecule_fock_rate
    from mmd.clusters import water_cluster
    rng = np.random.default_rng(seed)
    sizes = rng.integers(1, 9, size=nmol)
    geoms = [water_cluster(int(n), seed=10000 + k) for k, n in enumerate(sizes)]
    t0 = time.perf_counter()
    br = BatchRHF(geoms, "6-31g")
    t_setup = time.perf_counter() - t0
    # first-iteration density difference of every molecule (core guess)
    X, Core = br.X, br.Core
    FO = X.transpose(1, 2) @ Core @ X + torch.diag_embed(br.pad_shift)
    _, CO = br._eigh(FO)
    P1 = br._density(CO)
    dP = br._pack(P1)
    tun = autotune.autotune(br.ctx, dP.contiguous(), tol=br.acc2e)
    br.fock(P1)  # capture
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(reps):
        br.fock(P1)
    e1.record()
    torch.cuda.synchronize()
    t_b = e0.elapsed_time(e1) / 1e3 / reps
    # per-molecule launches on a subsample
    idx = np.arange(0, nmol, max(1, nmol // sample_per_molecule))[:sample_per_molecule]
    P1h = P1.cpu().numpy()
    rate_single = per_molecule_fock_rate([geoms[i] for i in idx], "6-31g",
                                         [P1h[i, :br.N[i], :br.N[i]] for i in idx])
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    E = br.run(conver=1e-8, polish=True)
    t_scf = time.perf_counter() - t0
    # parity: a seeded random subset of the molecules through the single-molecule path
    # (Molecule(...).RHF(direct=True), same convergence and polish) -- both energies
    # are exact to second order in their densities' error
    from mmd.molecule import Molecule
    pick = np.sort(np.random.default_rng(4242).choice(nmol, size=min(parity_sample, nmol), replace=False))
    dE = []
    for i in pick:
        e1 = Molecule(geoms[i], "6-31g").RHF(doPrint=False, direct=True, conver=1e-8, polish=True)
        dE.append(abs(float(E[i]) - float(e1)))
    return {"molecules": nmol, "basis": "6-31G", "n_water": "U{1..8}", "nbasis_total": int(br.N.sum()),
            "batched_fock_builds_per_s": nmol / t_b, "batched_ms_per_launch": 1e3 * t_b,
            "per_molecule_fock_builds_per_s": rate_single,
            "per_molecule_sample": int(len(idx)),
            "speedup": (nmol / t_b) / rate_single,
            "tuning": {"streams": tun.streams, "grids": tun.grids, "tiles": tun.tiles,
                       "build_ms_by_streams": tun.measured.get("build_ms_by_streams"),
                       "class_ms_by_tile": {k: {"tiles": v["tiles"], "total_ms": float(np.sum(v["class_ms"]))}
                                            for k, v in (tun.measured.get("class_ms_by_tile") or {}).items()}},
            "scf_time_s": t_scf, "scf_fock_launches": int(br.fock_builds),
            "converged": int(br.converged.sum()), "setup_s": t_setup,
            "mean_energy": float(np.mean(E)),
            "parity_vs_single_molecule": {"molecules": int(len(pick)), "max_abs_energy_diff_Eh": float(max(dE)),
                                          "sample": "seeded random subset (numpy default_rng(4242))",
                                          "energies": "FP64 polish build of each converged density, both paths"}}


def mixed_bench(n_water=32, thr=1e-5, conver=1e-8, seed=32):
    """Seeded (H2O)32 (4x4x2 lattice), 6-31G**, ~800 functions: direct RHF in FP64 and
    with quartets of Schwarz bound < thr in FP32.  Time to converge of both, and, in a
    second (checked) pass of each, the max |F - F_ref| of every iteration's Fock matrix
    against a from-scratch FP64 build on the same density (the FP64 pass gives the
    floor that incremental builds at acc2e = 1e-12 reach on their own)."""
    import numpy as np
    import torch
    from mmd.clusters import water_cluster
    from mmd.integrals import twoe
    from mmd.molecule import Molecule
    geom = water_cluster(n_water, seed=seed)
    out = {"workload": f"(H2O){n_water} 6-31G** direct RHF, seed {seed}", "fp32_below": thr, "conver": conver}
    for name, fp in (("fp64", 0.0), ("mixed", thr)):
        twoe.clear_context_cache()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        m = Molecule(geom, "6-31gss")
        E = float(m.RHF(doPrint=False, direct=True, fp32_below=fp, conver=conver))
        torch.cuda.synchronize()
        out[name] = {"energy": E, "time_to_converge_s": time.perf_counter() - t0, "iterations": int(m.iterations),
                     "converged": bool(m.is_converged)}
    out["nbasis"] = int(m.nbasis)
    out["energy_error_vs_fp64"] = out["mixed"]["energy"] - out["fp64"]["energy"]
    out["ttc_speedup"] = out["fp64"]["time_to_converge_s"] / out["mixed"]["time_to_converge_s"]
    for name, fp in (("fp64", 0.0), ("mixed", thr)):
        st = m.scf_begin(direct=True, fp32_below=fp, build=False)
        ctx, errs = m.context, []
        for step in range(m.maxiter):
            st.iterate()
            if step > 0:
                P = st.last_dP[0].contiguous()
                G = ctx.fock(P.view(-1), tol=m.scrTol, fp32_below=0.0).view(m.nbasis, m.nbasis)
                Fref = st.Core + 0.5 * (G + G.T)
                errs.append(float((st.F - Fref).abs().max().item()))
                if m.P_RMS < conver:
                    break
        out[name]["fock_max_error_per_iteration"] = errs
    # one full Fock build (converged density) in each precision, CUDA-event timed
    P = st.P.contiguous().view(-1)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for name, fp in (("fp64", 0.0), ("mixed", thr)):
        ctx.fock(P, tol=m.scrTol, fp32_below=fp)
        torch.cuda.synchronize()
        e0.record()
        for _ in range(3):
            ctx.fock(P, tol=m.scrTol, fp32_below=fp)
        e1.record()
        torch.cuda.synchronize()
        out[name]["full_fock_build_ms"] = e0.elapsed_time(e1) / 3
    out["fock_build_speedup"] = out["fp64"]["full_fock_build_ms"] / out["mixed"]["full_fock_build_ms"]
    return out


def _polished_energy(mol):
    """Energy of a finished Molecule(...).RHF's density from one non-incremental FP64
    Fock build (Molecule.polished_energy)."""
    return mol.polished_energy()


# FP32 threshold of the combined forms: quartets with Schwarz bound below 1e-3 in FP32.
# The final energy comes from an FP64 build (polish), so it is exact to second order
# in the density error whatever the threshold; measured on (H2O)16 6-31G** and 64
# (H2O)8 6-31G clusters, 1e-3 keeps the iteration counts of 1e-5 and every energy
# within 2e-12 Eh of the FP64 oracle, while moving more quartets off the FP64 pipe.
# The mixed-precision report on (H2O)32 (mixed_bench) keeps 1e-5.
COMBINED_FP32_BELOW = 1e-3
# the metric both arms report: the headline "RHF time-to-converge (1e-8 Eh) & Fock
# builds/s on 1 GB300, chosen form vs plain FP64", whose single number (value) is the
# plain FP64 Fock builds/s; the time-to-converge figures travel in the same line
METRIC = ("RHF time-to-converge (1e-8 Eh) & Fock builds/s on 1 GB300: chosen form vs plain FP64 "
          "[value: plain FP64 Fock builds/s, (H2O)16 6-31G** direct RHF, 20 iterations; "
          "time_to_converge_s, chosen_form]")
# time-to-converge figures of the benchmark molecule: best of this many end-to-end runs
# (fresh device context each), plain path and chosen form alike
TTC_RUNS = 2


def reference_energies_h2o8():
    """{seed: energy} of the reference's conventional RHF (conver 1e-12) on held-out
    (H2O)8 / 6-31G clusters (tests/golden/h2o8_631g_reference.json, made by
    tests/golden/make_golden_h2o8.py from the reference itself)."""
    path = os.path.join(REPO, "tests", "golden", "h2o8_631g_reference.json")
    if not os.path.exists(path):
        return {}
    with open(path) as f:
        return {int(m["seed"]): float(m["energy"]) for m in json.load(f)["molecules"]}


def combined_bench(nmol=64, thr=COMBINED_FP32_BELOW, conver=1e-8):
    """The three changes together on held-out seeded (H2O)8 clusters (6-31G): the plain
    FP64 GPU path (one Molecule(...).RHF(direct=True) after another, core guess) vs
    one BatchRHF over all molecules with FP32 below Schwarz thr and the learned guess
    (energies from an FP64 polish build), with two ablations (batched FP64 core
    guess, batched mixed core guess).  Times are wall clock from geometry strings to
    converged energies (set-up included).  Energy errors are against the reference's
    own conventional RHF energies (conver 1e-12) of the first eight molecules; the
    differences to the plain FP64 GPU path's polished energies cover all of them."""
    import numpy as np
    import torch
    from mmd import guess as G
    from mmd.batch import BatchRHF
    from mmd.clusters import water_cluster
    from mmd.molecule import Molecule
    geoms = [water_cluster(8, seed=900000 + k) for k in range(nmol)]
    Molecule(geoms[0], "6-31g").RHF(doPrint=False, direct=True, conver=conver)  # warm-up
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    Ep, itp, mols = [], [], []
    for g in geoms:
        m = Molecule(g, "6-31g")
        Ep.append(float(m.RHF(doPrint=False, direct=True, conver=conver)))
        itp.append(int(m.iterations))
        mols.append(m)
    torch.cuda.synchronize()
    t_plain = time.perf_counter() - t0
    Ep = np.array(Ep)
    Eo = np.array([_polished_energy(m) for m in mols])  # plain FP64 GPU path, polished
    ref = reference_energies_h2o8()  # the reference's own conventional RHF, conver 1e-12
    ridx = [k for k in range(nmol) if 900000 + k in ref]
    Er = np.array([ref[900000 + k] for k in ridx])

    def vs_ref(E):
        return float(np.abs(np.asarray(E)[ridx] - Er).max()) if ridx else None

    out = {"molecules": nmol, "workload": "(H2O)8 6-31G, seeds 900000+k (held out from training)",
           "conver": conver, "fp32_below": thr,
           "reference_energies": {"molecules": len(ridx), "source": "tests/golden/h2o8_631g_reference.json: the "
                                  "reference's conventional RHF (its compiled Cython doERIs), conver 1e-12"},
           "plain_fp64": {"time_to_converge_s": t_plain, "mean_iterations": float(np.mean(itp)),
                          "max_abs_energy_error_vs_reference": vs_ref(Ep),
                          "max_abs_energy_error_polished_vs_reference": vs_ref(Eo)}}
    net = G.DensityMLP.load()
    for name, fp, learned, cv, pf in (("batched_fp64_core", 0.0, False, conver, 0.0),
                                      ("batched_mixed_core", thr, False, conver, 0.0),
                                      ("batched_mixed_learned", thr, True, conver, 0.0),
                                      ("batched_mixed_learned_chosen_stopping_rule", thr, True, CHOSEN_CONVER,
                                       CHOSEN_POLISH_FP32_BELOW)):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        gs = [G.predict_density(net, Molecule(g, "6-31g")) for g in geoms] if learned else None
        br = BatchRHF(geoms, "6-31g", fp32_below=fp)
        E = br.run(conver=cv, guess=gs, polish=True, polish_fp32_below=pf)
        torch.cuda.synchronize()
        t = time.perf_counter() - t0
        out[name] = {"time_to_converge_s": t, "speedup_vs_plain": t_plain / t,
                     "mean_iterations": float(br.iterations.mean()), "converged": int(br.converged.sum()),
                     "max_abs_energy_error_vs_reference": vs_ref(E),
                     "max_abs_energy_diff_vs_plain_fp64_gpu_all": float(np.abs(E - Eo).max()),
                     "max_abs_energy_error_vs_reference_unpolished": vs_ref(br.energies_raw)}
        if learned:
            out[name]["reverted_to_core"] = int(br.reverted.sum())
    return out


def consumers_bench():
    """Wall times of the reference's consumers of the hot path on the GPU path:
    analytic forces (water 6-31G* distorted, (H2O)3 6-31G**), AO->MO + MP2
    ((H2O)4 6-31G), RT-TDHF Magnus4 steps (water 6-31G)."""
    import numpy as np
    import torch
    from mmd.clusters import water_cluster
    from mmd.molecule import Molecule
    from mmd.postscf import PostSCF
    from mmd.realtime import RealTime
    bent = "\n0 1\nO 0.0 -0.07 0.01\nH 0.80 0.62 0.03\nH -0.88 0.56 -0.02\n"
    out = {}

    def timed(fn):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        r = fn()
        torch.cuda.synchronize()
        return time.perf_counter() - t0, r

    for name, geom, basis in (("water_distorted", bent, "6-31gs"), ("(H2O)3", water_cluster(3, seed=4), "6-31gss")):
        mol = Molecule(geom, basis)
        mol.RHF(doPrint=False, conver=1e-10)
        mol.forces()  # warm
        t, _ = timed(mol.forces)
        out[f"forces_{name}_{basis}"] = {"s": t, "nbasis": int(mol.nbasis), "atoms": len(mol.atoms)}
    mol = Molecule(water_cluster(4, seed=4), "6-31g")
    mol.RHF(doPrint=False, conver=1e-10)
    PostSCF(mol).MP2()  # warm (library kernels load on first use)
    t, _ = timed(lambda: PostSCF(mol).MP2())
    out["ao2mo_mp2_(H2O)4_6-31g"] = {"s": t, "nbasis": int(mol.nbasis)}
    mol = Molecule(bent, "6-31g")

    def pulse(t):
        return np.exp(-((t - 1.0) ** 2) / 0.25)

    RealTime(mol, numsteps=5, stepsize=0.1, field=1e-3, pulse=pulse).Magnus4(direction="x")  # warm
    rt = RealTime(mol, numsteps=100, stepsize=0.1, field=1e-3, pulse=pulse)
    t, _ = timed(lambda: rt.Magnus4(direction="x"))
    out["rt_magnus4_water_6-31g"] = {"s_per_step": t / 100, "steps": 100, "nbasis": int(mol.nbasis)}
    return out


# The chosen form's stopping rule: ||P - P_old|| < 3e-5, then one polish build.  The
# polished energy E(P) = tr((H + F(P)) P) + E_nuc is stationary at the SCF solution,
# so its error is second order in the density error.  Measured on three (H2O)16
# 6-31G** geometries (seeds 16-18, learned guess; against the plain path's polished
# energy at conver 1e-10): stopping at 3e-4 / 1e-4 / 3e-5 / 1e-5 took 7 / 8-9 / 9 /
# 10-11 iterations with energy errors up to 6.3e-9 / 3.5e-10 / 6.1e-11 / 6.4e-12 Eh;
# 3e-5 keeps a 160-fold margin to the 1e-8 Eh target.  The same rule holds the
# held-out (H2O)8 within 1e-8 Eh of the reference's own energies
# (tests/test_gpu_reference_energies.py).  The plain path keeps the reference's rule
# (||dP|| < 1e-8 with the reference's first-order energy formula).  The iterations take
# FP32 below Schwarz 1e-1 (each such ERI off by at most 5e-7 x 1e-1; the density only
# has to reach 3e-5), the polish build FP32 below 1e-5 (at most 5e-12 per ERI).
# Measured on (H2O)16 (learned guess, 10 iterations; energy against the plain FP64
# path's polished energy at conver 1e-10): FP32 below 1e-3 / 1e-2 / 1e-1 / 1 in the
# iterations 0.419 / 0.413 / 0.392 / 0.378 s, energy error 0.9 / 1.0 / 1.1 / 11 e-11
# Eh; polish build FP32 below 0 / 1e-7 / 1e-6 / 1e-5 / 1e-4: 40.4 / 31.4 / 29.0 /
# 26.9 / 24.5 ms, energy error 0.3 / 0.6 / 0.5 / 0.09 / -2.5 e-11 Eh.
CHOSEN_FP32_BELOW = 1e-1
CHOSEN_CONVER = 3e-5
CHOSEN_POLISH_FP32_BELOW = 1e-5
# Eigensolver of the chosen form's iterations: the dense host solve of all N orbitals.
# The occupied-subspace solver (mmd.scf.OccupiedSubspace: Chebyshev-filtered subspace
# iteration on the GPU, 1.7 passes per iteration) measured slower at N = 400 (0.376
# against 0.359 s to converge): its ~25 small GEMMs and two host round trips per pass
# cost about what LAPACK's dsyevd takes for 400 x 400 (7 ms).  The line keeps it as an
# ablation.
CHOSEN_EIGENSOLVER = "dense"


def chosen_form_ttc(geom, ttc_plain, iters_plain, plain_mol, thr=CHOSEN_FP32_BELOW, conver=CHOSEN_CONVER,
                    polish_fp32_below=CHOSEN_POLISH_FP32_BELOW, learned=True, eigensolver=CHOSEN_EIGENSOLVER):
    """Time to converge of the benchmark molecule in the chosen form -- learned initial
    guess (the 6-31G** network), FP32 below Schwarz thr, stop at ||dP|| < conver, polish
    build -- against the plain FP64 path's time (measured just before, fresh context)
    and the plain FP64 GPU path's polished energy (the reference's own SCF at N = 400
    would take days; the plain path is pinned to the reference at the smaller sizes).
    ``learned=False, thr=0``: the plain path with the chosen form's stopping rule."""
    import torch
    from mmd import guess as G
    from mmd.integrals import twoe
    from mmd.molecule import Molecule
    E_oracle = plain_mol.polished_energy()
    net = G.network_for(Molecule(geom, "6-31gss")) if learned else None
    twoe.clear_context_cache()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    m = Molecule(geom, "6-31gss")
    P0 = G.predict_density(net, m) if learned else None
    E = float(m.RHF(doPrint=False, direct=True, fp32_below=thr, guess=P0, polish=True, conver=conver,
                    polish_fp32_below=polish_fp32_below, eigensolver=eigensolver))
    torch.cuda.synchronize()
    t = time.perf_counter() - t0
    form = ("learned guess + " if learned else "core guess + ") + \
        f"FP32 below {thr:g} + stop at ||dP|| < {conver:g} + polish (FP32 below {polish_fp32_below:g})" + \
        (" + occupied-subspace eigensolver" if eigensolver == "subspace" else "")
    sub = getattr(m, "subspace", None)
    subspace = None if sub is None else {"solves": sub.solves, "passes": sub.passes, "dense_fallbacks": sub.fallbacks,
                                         "block": sub.k, "degree": sub.degree, "tol": sub.tol}
    return {"form": form, "network": net.gb.name if learned else None,
            "time_to_converge_s": t,
            "iterations": int(m.iterations), "guess_reverted": bool(m.guess_reverted),
            "iterations_s": float(m.scf_time), "plain_iterations_s": float(plain_mol.scf_time),
            "speedup_vs_plain_fp64": ttc_plain / t, "plain_fp64_iterations": iters_plain,
            "energy": E, "energy_diff_vs_plain_fp64_gpu_polished": E - E_oracle, "subspace": subspace,
            "plain_fp64_energy_diff_vs_its_polished": float(plain_mol.energy) - E_oracle}


def fp64_roofline(class_ms, counts, builds, fp64_peak):
    """FP64-pipe roofline of the Fock build from per-class CUDA-event times and counters.

    Per class: ``issued`` = FP64 FLOPs the kernel issues (flop_model.pipe_flops:
    chunk passes, padded lanes and all), ``useful`` = the algorithm's own FLOPs (no
    recomputation or padding), ``model`` = the dense reference count; each as TFLOP/s
    and as a fraction of the measured DFMA peak.  The headline is the dominant
    class's issued rate."""
    import numpy as np
    from mmd import flop_model as F
    per = {}
    tot = {"issued": 0.0, "useful": 0.0, "model": 0.0}
    for c, ms, row in zip(F.CLASSES, class_ms, counts):
        if ms <= 0:
            continue
        fl = {"issued": F.pipe_flops(c, row), "useful": F.useful_flops(c, row),
              "model": F.class_flops(c, row[2], row[0])}
        for k in tot:
            tot[k] += fl[k]
        t = ms / 1e3
        per["%d%d%d%d" % c] = {"ms_per_build": float(ms) / builds, "kernel": F.fock_kernel(c),
                               **{f"{k}_frac": fl[k] / t / 1e12 / fp64_peak for k in fl}}
    dom = int(np.argmax(class_ms))
    c = F.CLASSES[dom]
    key = "%d%d%d%d" % c
    row = counts[dom]
    issued = F.pipe_flops(c, row)
    t = class_ms[dom] / 1e3
    achieved = issued / t / 1e12
    kern = "k_fock_warp<MDW_%s,double>" % key if F.fock_kernel(c) == "warp" else "k_fock<MD_%s,double>" % key
    T = float(np.sum(class_ms)) / 1e3
    return {"bound": "fp64", "kernel": kern, "class": key, "achieved": achieved, "peak": fp64_peak,
            "unit": "TFLOP/s", "frac": achieved / fp64_peak,
            "flops": "issued FP64 FLOPs (2 per DFMA, 1 per DMUL/DADD) counted from the code and the build's "
                     "counters; excludes the FP64 instructions inside CUDA's exp (asymptotic Boys, L >= 5)",
            "flops_per_launch": issued / builds, "launch_ms": float(class_ms[dom]) / builds,
            "useful_frac": F.useful_flops(c, row) / t / 1e12 / fp64_peak,
            "model_frac": F.class_flops(c, row[2], row[0]) / t / 1e12 / fp64_peak,
            "peak_source": "live DFMA probe mmdg_measure_peaks (MEASURED_PEAKS.json has no FP64 figure)",
            "all_classes": {"fock_build_ms": float(np.sum(class_ms)) / builds,
                            "issued_frac": tot["issued"] / T / 1e12 / fp64_peak,
                            "useful_frac": tot["useful"] / T / 1e12 / fp64_peak,
                            "model_frac": tot["model"] / T / 1e12 / fp64_peak},
            "per_class": per}


# ------------------------------------------------------------------------------ GPU arm
def gpu_arm(args):
    import numpy as np
    import torch
    rank, world, local = _env()
    torch.cuda.set_device(local)
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl")
    sys.path.insert(0, PKG)
    from mmd import _native, flop_model
    from mmd.clusters import water_cluster
    from mmd.integrals.fock import formPT
    from mmd.molecule import Molecule

    if args.n_water != WORKLOAD["n_water"]:  # smaller clusters for profiling captures
        WORKLOAD.update(n_water=args.n_water, workload=f"(H2O){args.n_water} 6-31G** direct RHF", nbasis=25 * args.n_water)
    geom = water_cluster(WORKLOAD["n_water"], seed=WORKLOAD["seed"])
    fp32 = args.fp32_below
    # ---------------- warm-up SCF
    mol = Molecule(geom, "6-31gss")
    N = mol.nbasis
    st = mol.scf_begin(direct=True, acc2e=WORKLOAD["schwarz"], fp32_below=fp32)
    for _ in range(args.warmup + 1):
        st.iterate()
    # ---------------- timed: iterations 1..K of a fresh SCF
    st = mol.scf_begin(direct=True, acc2e=WORKLOAD["schwarz"], fp32_below=fp32, build=False)
    st.iterate()  # iteration 0: core-Hamiltonian diagonalisation, no Fock build
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float64, device="cuda")
    dens = []
    clocks = ClockSampler(local)
    clocks.start()
    if world > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    wall0 = time.perf_counter()
    for k in range(args.steps):
        flush.zero_()
        ev[k][0].record()
        st.iterate()
        ev[k][1].record()
        dens.append(st.last_dP)
    torch.cuda.synchronize()
    wall = time.perf_counter() - wall0
    if world > 1:
        torch.distributed.barrier()
    clk = clocks.stop()
    step_ms = [a.elapsed_time(b) for a, b in ev]
    t_dev = sum(step_ms) / 1e3
    t_dev = max_over_ranks(t_dev, "cuda")
    builds = args.steps
    value = replica_throughput(world, builds, t_dev)
    # ---------------- per-class profile: the same K density differences again, each
    # class kernel timed alone by CUDA events (one stream), with its quartet counts
    ctx = mol.context
    class_ms = np.zeros(len(flop_model.CLASSES))
    counts = np.zeros((len(flop_model.CLASSES), _native.NCOUNT))
    L2flush = flush
    for P_, Po_ in dens:
        L2flush.zero_()
        _, ms, cnt = ctx.fock_timed((P_ - Po_).contiguous().view(-1), tol=WORKLOAD["schwarz"], fp32_below=fp32)
        class_ms += ms.astype(np.float64)
        counts += cnt.astype(np.float64)
    fq_per_build = float(counts[:, 0].sum()) / builds
    # ---------------- FP64 roofline: FLOPs the kernels issue (counted from the code's
    # structure and the build's counters; ncu's DFMA/DMUL/DADD counters are the
    # cross-check), the algorithm's useful FLOPs and the dense reference model
    fp64_peak, fp32_peak = _native.measure_peaks(ctx)
    roofline = fp64_roofline(class_ms, counts, builds, fp64_peak)
    roofline["fp32_peak"] = fp32_peak
    # the FP64 tensor cores beside the DFMA pipe (why the transforms stay on DFMA)
    roofline["fp64_pipes"] = _native.measure_fp64_pipes(ctx, 16)
    if WORKLOAD["n_water"] == 16:
        key = roofline["class"]
        roofline["traffic"] = DRAM_BYTES_PER_LAUNCH.get(key)
        roofline["fp64_pipe_busy_ncu"] = FP64_PIPE_BUSY.get(key)
    else:
        roofline["traffic"] = None
    build_ms = float(class_ms.sum()) / builds  # class kernels timed one after another
    # ---------------- e2e through formPT with host arrays
    Ph = [(a.cpu().numpy(), b.cpu().numpy()) for a, b in dens]
    screen = mol.screen
    formPT(Ph[0][0], Ph[0][1], mol.bfs, N, screen, WORKLOAD["schwarz"])  # context / screen already cached
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for P, Po in Ph:
        G = formPT(P, Po, mol.bfs, N, screen, WORKLOAD["schwarz"])
    t_e2e = time.perf_counter() - t0
    del G
    e2e = {"value": world * len(Ph) / t_e2e, "unit": "Fock builds/s", "api": "mmd.integrals.fock.formPT (host arrays)",
           "h2d_bytes_per_step": N * N * 8, "d2h_bytes_per_step": N * N * 8}
    # ---------------- time to converge through Molecule(...).RHF (fresh device context),
    # best of TTC_RUNS runs for the plain path and for the chosen form alike
    ttc, E, iters = None, None, None
    if not args.no_ttc:
        from mmd.integrals import twoe
        for _ in range(TTC_RUNS):
            twoe.clear_context_cache()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            m_ = Molecule(geom, "6-31gss")
            E_ = float(m_.RHF(doPrint=False, direct=True, fp32_below=fp32))
            t_ = time.perf_counter() - t0
            if ttc is None or t_ < ttc:
                ttc, E, iters, m2 = t_, E_, int(m_.iterations), m_
    chosen = None
    if not args.no_ttc and rank == 0 and fp32 == 0.0:
        try:
            runs = [chosen_form_ttc(geom, ttc, iters, m2) for _ in range(TTC_RUNS)]
            chosen = min(runs, key=lambda r: r["time_to_converge_s"])
            chosen["runs"] = TTC_RUNS
            # ablations: the chosen form under the reference's stopping rule, and the
            # plain FP64 path under the chosen form's stopping rule
            keep = ("form", "time_to_converge_s", "iterations", "speedup_vs_plain_fp64",
                    "energy_diff_vs_plain_fp64_gpu_polished")
            a = chosen_form_ttc(geom, ttc, iters, m2, conver=1e-8, polish_fp32_below=0.0)
            chosen["at_reference_stopping_rule"] = {k: a[k] for k in keep}
            a = chosen_form_ttc(geom, ttc, iters, m2, eigensolver="subspace")
            chosen["with_subspace_eigensolver"] = {k: a[k] for k in keep + ("subspace",)}
            b = chosen_form_ttc(geom, ttc, iters, m2, thr=0.0, polish_fp32_below=0.0, learned=False,
                                eigensolver="dense")
            chosen["plain_fp64_at_chosen_stopping_rule"] = {k: b[k] for k in keep}
        except Exception as e:  # reported, never required for the headline
            chosen = {"error": str(e)[:300]}
    # ---------------- CPU baseline (rank 0, N = 1)
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        npair = N * (N + 1) // 2
        try:
            cb = run_cpu_sample(npair * (npair + 1) // 2, fq_per_build, steps=2, warmup=1)
            cpu = {"value": cb["builds_per_s"], "unit": "Fock builds/s", "cores": cb["cores"], "kind": cb["kind"],
                   "sample": cb["sample"], "t_build_1core_s": cb["t_build_1core_s"],
                   "quartets_per_s_1core": cb["quartets_per_s_1core"], "anchor": cb.get("anchor")}
        except Exception as e:  # the baseline is reported, never required
            cpu = {"value": None, "error": str(e)[:300]}
    # our kernels per Fock build: k_shell_dmax, k_screen, one k_fock per class and
    # precision, and k_fock_update of the SCF step
    launches_per_build = 3 + len(flop_model.CLASSES) * (2 if fp32 > 0 else 1)
    batched = mixed = combined = None
    if rank == 0 and not args.no_batch:
        try:
            batched = batched_bench()
        except Exception as e:  # reported, never required for the headline
            batched = {"error": str(e)[:300]}
    if rank == 0 and not args.no_mixed:
        try:
            mixed = mixed_bench()
        except Exception as e:
            mixed = {"error": str(e)[:300]}
    consumers = None
    if rank == 0 and args.consumers:
        try:
            consumers = consumers_bench()
        except Exception as e:
            consumers = {"error": str(e)[:300]}
    if rank == 0 and not args.no_combined:
        try:
            combined = combined_bench()
        except Exception as e:
            combined = {"error": str(e)[:300]}
    line = {
        "metric": METRIC,
        "value": value, "unit": "Fock builds/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1e3 * t_dev / builds, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f64" if fp32 == 0 else "f64+f32", "data": "synthetic (seeded cluster geometry)",
        "config": dict(WORKLOAD, fp32_below=fp32, l2="flushed between steps (512 MB write)",
                       fq_per_build=fq_per_build, eris_per_s=fq_per_build * value / world,
                       parallelism="replicas" if world > 1 else "single GPU"),
        "e2e": e2e, "time_to_converge_s": ttc, "ttc_runs": TTC_RUNS, "scf_iterations": iters, "energy": E,
        "chosen_form": chosen,
        "roofline": roofline, "cpu_baseline": cpu, "clocks": clk,
        "gpu_launches": launches_per_build * builds, "wall_s": wall,
        "step_breakdown_ms": {"step": 1e3 * t_dev / builds, "fock_class_kernels_one_stream": build_ms,
                              "note": "the timed steps run the class kernels on 8 concurrent streams; the "
                                      "per-class profile replays the same densities on one stream"},
        "batched": batched, "mixed_precision": mixed, "combined_form": combined, "consumers": consumers,
        "class_ms_per_build": {"%d%d%d%d" % c: float(x) / builds for c, x in zip(flop_model.CLASSES, class_ms)},
        "class_counts_per_build": {"%d%d%d%d" % c: [float(v) / builds for v in row]
                                   for c, row in zip(flop_model.CLASSES, counts)},
    }
    if rank == 0:
        print(json.dumps(line))
    if world > 1:
        torch.distributed.destroy_process_group()


# ------------------------------------------------------------------------------ reference arm
def reference_arm(args):
    rank, world, _ = _env()
    if rank != 0:
        return
    npair = 400 * 401 // 2
    if FQ_PER_BUILD is None:
        print(json.dumps({"impl": "reference", "unavailable": "survivor count of the workload not yet recorded"}))
        return
    cb = run_cpu_sample(npair * (npair + 1) // 2, FQ_PER_BUILD, steps=args.steps, warmup=args.warmup)
    v = cb["builds_per_s"]
    line = {"impl": "reference", "metric": METRIC, "value": v,
            "unit": "Fock builds/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": 1e3 / v, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic (seeded cluster geometry)", "config": dict(WORKLOAD),
            "cpu_baseline": {"value": v, "unit": "Fock builds/s", "cores": cb["cores"], "kind": cb["kind"],
                             "sample": cb["sample"], "t_build_1core_s": cb["t_build_1core_s"],
                             "quartets_per_s_1core": cb["quartets_per_s_1core"], "anchor": cb.get("anchor")},
            "e2e": {"value": v, "unit": "Fock builds/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--fp32-below", type=float, default=0.0, help="Schwarz bound below which quartets run in FP32")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU-baseline sample")
    ap.add_argument("--no-ttc", action="store_true", help="skip the time-to-converge run")
    ap.add_argument("--no-batch", action="store_true", help="skip the 1024-molecule batched sub-benchmark")
    ap.add_argument("--no-mixed", action="store_true", help="skip the (H2O)32 mixed-precision sub-benchmark")
    ap.add_argument("--no-combined", action="store_true", help="skip the learned+batched+mixed sub-benchmark")
    ap.add_argument("--consumers", action="store_true", help="also time forces, MP2 and RT-TDHF")
    ap.add_argument("--n-water", type=int, default=16, help="cluster size (16 = the benchmark workload)")
    ap.add_argument("--cpu-sample", metavar="SPEC")
    ap.add_argument("--cores", type=int, default=None)
    args = ap.parse_args()
    if args.cpu_sample:
        cpu_sample(args.cpu_sample, args.cores or os.cpu_count(), args.steps, args.warmup)
    elif args.impl == "reference":
        reference_arm(args)
    else:
        gpu_arm(args)


if __name__ == "__main__":
    main()
