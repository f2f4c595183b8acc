#!/usr/bin/env python
"""Benchmark: two-site gates/s at chi=256 (40-qubit Haar brickwork, depth 20).

Workload (one "step"): the full 390-gate circuit from |0...0>, 40 qubits,
brickwork of Haar-random 4x4 unitaries (seeded QR of complex Gaussians), chi_max
256, eps_bond 1e-8, complex64 -- run through the AdaptiveMPS API of this package
in its device-resident mode (``device_resident=True``: bond dimensions stay on
the device, no host synchronisation between batches); ``--host-sync`` times the
host-synchronised mode instead, and the line reports the other mode beside it.

Lines printed (rank 0, one JSON object):
  value    gates/s with gate matrices already resident in HBM (device events)
  e2e      gates/s through the public API with the gates in pinned host memory
           (host->device copies and the device->host result read inside the timing)
  roofline the dominant kernel, from the library's live per-stage CUDA events
  cpu_baseline  the reference's complex64 two-site update on this host's cores
           (PyTorch-CPU port with the reference's own library calls), bounded sample
  plain_gpu     the reference call sequence on this GPU with torch complex64
           contraction + torch.linalg.svd (cuSOLVER), for the plain-form comparison
  learned  the host-synchronised pipeline with the learned rank predictor sizing
           each gate's eigensolver (weights shipped in atlasq_gb300/data/)
  graph_replay  the same circuit captured once as a CUDA graph and replayed
  fidelity_vs_fp64  |<psi|psi_fp64>|^2 of each arm's final state against this
           package's complex128 run of the same circuit

``--impl reference`` times the CPU port of the reference path instead.
Multi-GPU (torchrun): independent replicas per rank, no collective on the data
path ("scaling": "weak").
"""
import argparse
import ctypes
import json
import math
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np
import torch

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

N_QUBITS, DEPTH, CHI, EPS, SEED = 40, 20, 256, 1e-8, 1234
METRIC = "2-site gates/s at chi=256 (40q Haar brickwork depth 20, eps 1e-8)"
WORKLOAD = "40-qubit Haar brickwork depth 20 (390 two-site gates), chi_max=256, eps_bond=1e-8, complex64"
L2_BYTES = 129 * 1024 * 1024
PORT_NOTE = ("; PyTorch-CPU port of the reference's complex64 apply_two_site_gate (einsum, torch.linalg.svd, "
             "float32 rank rule), all host threads; measured at 0.92-1.09x the reference's own time on one CPU")


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), float(p["bf16_tflops"]), "measured"
    except Exception:
        return 6800.0, 1900.0, "fallback"


class ClockSampler:
    """nvidia-smi samples during the timed region (SM clock, throttle reasons)."""

    def __init__(self, index):
        self.index = index
        self.samples = []
        self.proc = None
        self.thread = None

    def start(self):
        q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except Exception:
            self.proc = None
            return
        self.thread = threading.Thread(target=self._read, daemon=True)
        self.thread.start()

    def _read(self):
        for line in self.proc.stdout:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) >= 8:
                self.samples.append(parts)

    def stop(self):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()
        if self.thread is not None:
            self.thread.join(timeout=2)
        sm = []
        mx = None
        reasons = set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for p in self.samples:
            try:
                sm.append(float(p[0]))
                mx = float(p[1])
            except ValueError:
                continue
            for nm, v in zip(names, p[4:8]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx,
                "reasons": sorted(reasons), "samples": len(sm)}


def config_of(n_replicas):
    """The workload description both arms report (same keys, same values)."""
    gates = (DEPTH + 1) // 2 * (N_QUBITS // 2) + DEPTH // 2 * (N_QUBITS // 2 - 1)  # even layers 20, odd 19
    return {"workload": WORKLOAD, "gates_per_step": gates, "parallelism": f"replicas x{n_replicas}"}


def make_circuit():
    from atlasq_gb300.circuits import haar_brickwork
    return haar_brickwork(N_QUBITS, DEPTH, seed=SEED)


RESIDENT = True  # the headline runs AdaptiveMPS(device_resident=True); --host-sync switches to the host-synchronised mode


def run_ours(ops, device, dtype=torch.complex64, resident=None):
    import atlasq_gb300 as aq
    pol = aq.DTypePolicy(default=dtype)
    m = aq.AdaptiveMPS(N_QUBITS, bond_dim=1, eps_bond=EPS, chi_max_per_bond=CHI, device=device,
                       dtype=dtype, dtype_policy=pol, device_resident=RESIDENT if resident is None else resident)
    for _, q, U in ops:
        m.apply_two_site_gate(q, U)
    m.flush()
    return m


def mps_overlap(ta, tb):
    """<a|b> with the package GEMMs (left environment sweep)."""
    from atlasq_gb300 import ops as o
    E = torch.ones(1, 1, dtype=torch.complex128, device=ta[0].device)
    for A, B in zip(ta, tb):
        A = A.to(torch.complex128).contiguous()
        B = B.to(torch.complex128).contiguous()
        la, _, ra = A.shape
        lb, _, rb = B.shape
        M = o.cgemm(E, B.reshape(lb, 2 * rb))                     # [la, 2rb]
        E = o.cgemm(A.reshape(2 * la, ra), M.reshape(2 * la, rb), opA="C", opB="N")
    return complex(E[0, 0].item())


def plain_gpu_circuit(ops, device):
    """Reference call sequence (adaptive_mps.py:182-308) with torch on the GPU:
    einsum contraction (mps_complex.py:343-368), torch.linalg.svd (cuSOLVER),
    the rank rule with its host syncs (truncation.py:21-83), U*S | Vh split."""
    from atlasq_gb300.truncation import choose_rank_from_sigma
    tensors = [torch.zeros(1, 2, 1, dtype=torch.complex64, device=device) for _ in range(N_QUBITS)]
    for t in tensors:
        t[0, 0, 0] = 1
    for _, i, U in ops:
        A, B = tensors[i], tensors[i + 1]
        li, ri, rj = A.shape[0], A.shape[2], B.shape[2]
        psi = torch.einsum("lpr,rqj->lpqj", A, B).permute(1, 2, 0, 3).reshape(4, li * rj)
        X = (U @ psi).reshape(2, 2, li, rj).permute(2, 0, 1, 3).reshape(li * 2, 2 * rj)
        Uu, S, Vh = torch.linalg.svd(X, full_matrices=False)
        E = (S * S).cumsum(0)
        total = E[-1]
        thresh = (1.0 - EPS ** 2) * total
        k = min(int(torch.searchsorted(E, thresh).item()) + 1, S.numel(), CHI)
        _ = float(torch.sqrt(torch.clamp(total - E[k - 1], min=0)).item())
        tensors[i] = (Uu[:, :k] * S[:k]).reshape(li, 2, k)
        tensors[i + 1] = Vh[:k].reshape(k, 2, rj)
    return tensors


def cpu_port_circuit(ops, time_cap=None):
    """The reference's complex64 two-site update on the host cores: the
    PyTorch-CPU port (same library calls as adaptive_mps.py:182-308: einsum
    contraction, torch.linalg.svd, float32 rank rule).  Returns gates done, seconds."""
    from oracle.torch_port import TorchPortMPS
    torch.set_num_threads(os.cpu_count() or 1)
    m = TorchPortMPS(N_QUBITS, eps_bond=EPS, chi_max=CHI)
    t0 = time.perf_counter()
    done = 0
    for _, q, U in ops:
        m.apply_two_site_gate(q, U)
        done += 1
        if time_cap is not None and time.perf_counter() - t0 > time_cap:
            break
    return done, time.perf_counter() - t0


def dist_init():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if ws > 1:
        import torch.distributed as dist
        backend = "nccl" if torch.cuda.is_available() else "gloo"
        dist.init_process_group(backend=backend)
        return dist, ws, rank, local
    return None, 1, 0, local


def barrier(dist, device=None):
    if dist is not None:
        if device is not None and dist.get_backend() == "nccl":
            dist.barrier(device_ids=[device.index])
        else:
            dist.barrier()


def max_over_ranks(dist, x, device):
    if dist is None:
        return x
    t = torch.tensor([x], dtype=torch.float64, device=device if dist.get_backend() == "nccl" else "cpu")
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def reference_arm(args, dist, ws, rank):
    """--impl reference: the reference path's CPU implementation (oracle port) on host cores."""
    if rank != 0:
        return
    ops = make_circuit()
    cores = os.cpu_count() or 1
    cap = float(os.environ.get("AGB_REF_STEP_CAP_S", "45"))
    for _ in range(min(args.warmup, 1)):
        cpu_port_circuit(ops[:40])
    total_g, total_t = 0, 0.0
    for _ in range(args.steps):
        g, t = cpu_port_circuit(ops, time_cap=cap)
        total_g += g
        total_t += t
    v = total_g / total_t
    sample = ("full 390-gate circuit per step" if total_g == 390 * args.steps else
              f"{total_g} gates over {args.steps} steps (each step capped at {cap:.0f} s)")
    line = {"metric": METRIC, "value": v, "unit": "gates/s", "n_gpus": args.gpus, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": 1000.0 * total_t / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "complex64", "data": "synthetic",
            "impl": "reference", "config": config_of(args.gpus),
            "cpu_baseline": {"value": v, "unit": "gates/s", "cores": cores, "kind": "port",
                             "sample": sample + PORT_NOTE},
            "e2e": {"value": v, "unit": "gates/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def _timed(fn, device):
    torch.cuda.synchronize()
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    out = fn()
    e.record()
    e.synchronize()
    return out, s.elapsed_time(e)


def secondary_workload(args):
    """One JSON line for a secondary workload (1 GPU):
    batch256  256 HEA instances (n ~ U{16..48}, chi_max in {64,128,256}, 10 layers, eps 1e-8)
              advanced together by MPSBatch; gates/s over all instances
    sample50  50-qubit chi=256 Haar brickwork depth 16: 100,000 Philox shots, then 49 <Z_i Z_i+1>
              and 50 <X_i>; shots/s (the state build is untimed)
    hea64     64-qubit HEA, 12 layers of RY RZ + CZ ladder, chi_max 512, eps 1e-8; gates/s"""
    import atlasq_gb300 as aq
    from atlasq_gb300 import _lib
    from atlasq_gb300.circuits import haar_brickwork, hea_circuit
    lib = _lib.load()
    device = torch.device("cuda", 0)
    torch.cuda.set_device(device)
    flush_buf = torch.empty(2 * L2_BYTES, dtype=torch.uint8, device=device)
    line = {"n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "complex64", "data": "synthetic"}
    if args.workload == "batch256":
        rng = np.random.default_rng(2024)
        specs = []
        for b in range(256):
            n = int(rng.integers(16, 49))
            chi = int(rng.choice([64, 128, 256]))
            ops = [(k, q, U.to(device)) for k, q, U in hea_circuit(n, 10, seed=50000 + b)]
            specs.append((n, chi, ops))
        ngates = sum(sum(1 for op in o if op[0] == "2q") for _, _, o in specs)

        def fresh(resident):
            return [aq.AdaptiveMPS(n, bond_dim=1, eps_bond=1e-8, chi_max_per_bond=chi, device=device,
                                   device_resident=resident) for n, chi, _ in specs]
        # (1) host-synchronised batches (one ranks read-back per round)
        insts = fresh(False)
        flush_buf.zero_()
        batch, ms_sync = _timed(lambda: aq.MPSBatch(insts).run([o for _, _, o in specs]), device)
        ref_dims = [list(m.bond_dims) for m in insts]
        # (2) device-resident, the whole 256-instance circuit captured as one CUDA graph
        insts = fresh(True)
        t0 = time.perf_counter()
        cap = aq.MPSBatch(insts).capture([o for _, _, o in specs])
        torch.cuda.synchronize()
        capture_s = time.perf_counter() - t0
        for _ in range(args.warmup):
            cap.replay()
        torch.cuda.synchronize()
        launches0 = lib.agb_launch_count()
        tot = 0.0
        for _ in range(args.steps):
            flush_buf.zero_()
            torch.cuda.synchronize()
            s_, e_ = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            s_.record(cap.stream)
            cap.replay()
            e_.record(cap.stream)
            e_.synchronize()
            tot += s_.elapsed_time(e_)
        ms = tot / args.steps
        cap.finish()
        same = sum(1 for m, d in zip(insts, ref_dims) if list(m.bond_dims) == d)
        line.update({"metric": "2-site gates/s, 256 HEA instances advanced together", "value": ngates / (ms / 1e3),
                     "unit": "gates/s", "ms_per_step": ms,
                     "gpu_launches": cap.kernels_per_replay,
                     "config": {"workload": "256 HEA instances, n~U{16..48}, chi_max in {64,128,256}, 10 layers, eps 1e-8",
                                "gates_per_step": ngates, "rounds_per_step": len(cap.rounds),
                                "execution": "device-resident, whole circuit as one CUDA graph (replay timed)",
                                "max_bond": max(max(m.bond_dims) for m in insts)},
                     "host_synchronised": {"value": ngates / (ms_sync / 1e3), "unit": "gates/s",
                                           "rounds": batch.rounds},
                     "capture_seconds": capture_s,
                     "instances_with_identical_bond_dims": same})
    elif args.workload == "sample50":
        from atlasq_gb300.sampling import right_canonical_copy, sample_tensors
        ops = [(k, q, U.to(device)) for k, q, U in haar_brickwork(50, 16, seed=77)]
        m = aq.AdaptiveMPS(50, bond_dim=1, eps_bond=1e-8, chi_max_per_bond=256, device=device)
        for _, q, U in ops:
            m.apply_two_site_gate(q, U)
        m.flush()
        Z = torch.tensor([[1, 0], [0, -1]], dtype=torch.complex64)
        X = torch.tensor([[0, 1], [1, 0]], dtype=torch.complex64)
        obs = [{i: Z, i + 1: Z} for i in range(49)] + [{i: X} for i in range(50)]
        shots = 100000

        def one():
            flush_buf.zero_()
            def work():
                ts = right_canonical_copy(m)
                bits = sample_tensors(ts, shots, seed=5)
                vals = aq.local_expectations(m, obs)
                return bits, vals
            return _timed(work, device)
        for _ in range(args.warmup):
            one()
        launches0 = lib.agb_launch_count()
        tot = 0.0
        for _ in range(args.steps):
            (bits, vals), ms = one()
            tot += ms
        ms = tot / args.steps
        launches = (lib.agb_launch_count() - launches0) // max(args.steps, 1)
        # sampling alone
        ts = right_canonical_copy(m)
        torch.cuda.synchronize()
        _, ms_s = _timed(lambda: sample_tensors(ts, shots, seed=5), device)
        _, ms_e = _timed(lambda: aq.local_expectations(m, obs), device)
        chis = [t.shape[0] for t in ts] + [1]
        flops = sum(8.0 * 2 * shots * chis[i] * chis[i + 1] for i in range(50))  # complex MACs: L[ns,l] x T[l,2r]
        line.update({"metric": "shots/s (100k Philox shots + 99 local expectations, 50q chi=256)",
                     "value": shots / (ms / 1e3), "unit": "shots/s", "ms_per_step": ms, "gpu_launches": launches,
                     "config": {"workload": "50-qubit Haar brickwork depth 16, chi_max 256; 100,000 shots; 49 ZZ + 50 X",
                                "max_bond": max(chis)},
                     "parts_ms": {"right_canonicalise+sample": ms_s, "expectations": ms_e},
                     "sampling_tflops": flops / (ms_s / 1e3) / 1e12,
                     "zz0": vals[0].real, "x0": vals[49].real})
    else:
        ops = [(k, q, U.to(device)) for k, q, U in hea_circuit(64, 12, seed=64)]
        ngates = sum(1 for op in ops if op[0] == "2q")

        def one():
            m = aq.AdaptiveMPS(64, bond_dim=1, eps_bond=1e-8, chi_max_per_bond=512, device=device)
            flush_buf.zero_()

            def work():
                for k, q, U in ops:
                    (m.apply_two_site_gate if k == "2q" else m.apply_single_qubit_gate)(q, U)
                m.flush()
                return m
            return _timed(work, device)
        for _ in range(args.warmup):
            one()
        lib.agb_prof_begin(200000)
        tot = 0.0
        for _ in range(args.steps):
            m, ms = one()
            tot += ms
        ms = tot / args.steps
        ms_st = (ctypes.c_double * 16)()
        cnt_st = (ctypes.c_int * 16)()
        _lib.check(lib.agb_prof_end(ms_st, cnt_st, 16), "prof_end")
        line.update({"metric": "2-site gates/s, 64q HEA 12 layers chi=512", "value": ngates / (ms / 1e3),
                     "unit": "gates/s", "ms_per_step": ms,
                     "config": {"workload": "64-qubit HEA, 12 layers RY RZ + CZ ladder, chi_max 512, eps 1e-8",
                                "gates_per_step": ngates, "max_bond": max(m.bond_dims)},
                     "stage_ms_per_step": {nm: round(ms_st[i] / args.steps, 3) for i, nm in enumerate(_lib.STAGES)}})
    print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-plain", action="store_true")
    ap.add_argument("--resident", action="store_true",
                    help="AdaptiveMPS(device_resident=True), no host synchronisation between batches: the default")
    ap.add_argument("--host-sync", action="store_true",
                    help="run AdaptiveMPS(device_resident=False): ranks read back after every batch")
    ap.add_argument("--workload", default="brickwork40", choices=["brickwork40", "batch256", "sample50", "hea64"],
                    help="brickwork40 is the headline; the others are the secondary workloads")
    ap.add_argument("--no-learned", action="store_true", help="skip the learned-rank arm")
    ap.add_argument("--no-graph", action="store_true", help="skip the CUDA-graph replay line")
    ap.add_argument("--two-stage", action="store_true",
                    help="use the two-stage tridiagonalisation (band reduction + bulge chasing) instead of the "
                         "one-stage cluster kernel, for comparison")
    args = ap.parse_args()
    if args.gpus > 1 and "WORLD_SIZE" not in os.environ:
        # one process per GPU: relaunch this command under torch.distributed.run
        cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", f"--nproc-per-node={args.gpus}",
               "--master-addr", "127.0.0.1", "--master-port", os.environ.get("MASTER_PORT", "29511"),
               os.path.abspath(__file__)] + sys.argv[1:]
        sys.exit(subprocess.call(cmd))
    global RESIDENT
    RESIDENT = not args.host_sync
    if args.workload != "brickwork40" and args.impl == "ours":
        secondary_workload(args)
        return

    dist, ws, rank, local = dist_init()
    if args.impl == "reference":
        reference_arm(args, dist, ws, rank)
        if dist is not None:
            dist.destroy_process_group()
        return

    import atlasq_gb300 as aq
    from atlasq_gb300 import _lib
    lib = _lib.load()
    if args.two_stage:
        _lib.check(lib.agb_set_tridiag_stages(0), "set_tridiag_stages")
    device = torch.device("cuda", local)
    torch.cuda.set_device(device)
    ops_host = make_circuit()
    ngates = len(ops_host)
    ops_dev = [(k, q, U.to(device)) for k, q, U in ops_host]
    ops_pinned = [(k, q, U.pin_memory()) for k, q, U in ops_host]
    flush_buf = torch.empty(2 * L2_BYTES, dtype=torch.uint8, device=device)

    for _ in range(max(args.warmup, 3) if args.warmup > 0 else 0):
        run_ours(ops_dev, device)
    torch.cuda.synchronize()

    # ---------------------------------------------------------------- timed region (value)
    lib.agb_prof_begin(200000)
    launches0 = lib.agb_launch_count()
    sampler = ClockSampler(local)
    sampler.start()
    barrier(dist, device)
    torch.cuda.synchronize()
    total_ms = 0.0
    last = None
    for _ in range(args.steps):
        flush_buf.zero_()  # L2 flush between timed iterations (untimed)
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        last = run_ours(ops_dev, device)
        e.record()
        e.synchronize()
        total_ms += s.elapsed_time(e)
    torch.cuda.synchronize()
    barrier(dist, device)
    clocks = sampler.stop()
    launches = lib.agb_launch_count() - launches0
    ms_st = (ctypes.c_double * 16)()
    cnt_st = (ctypes.c_int * 16)()
    _lib.check(lib.agb_prof_end(ms_st, cnt_st, 16), "prof_end")
    stage_ms = {name: ms_st[i] / args.steps for i, name in enumerate(_lib.STAGES)}
    total_ms = max_over_ranks(dist, total_ms, device)
    ms_per_step = total_ms / args.steps
    value = ngates * ws / (ms_per_step / 1000.0)

    # ---------------------------------------------------------------- e2e (host buffers)
    torch.cuda.synchronize()
    e2e_ms = 0.0
    for _ in range(args.steps):
        flush_buf.zero_()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        m = run_ours(ops_pinned, device)
        res = [t.cpu() for t in m.tensors]  # device->host read of the step's result: every site tensor
        torch.cuda.synchronize()
        e2e_ms += (time.perf_counter() - t0) * 1000.0
    e2e_ms = max_over_ranks(dist, e2e_ms, device) / args.steps
    # per step: gate matrices (16 complex64) + two descriptor uploads per gate (32 int64 each);
    # back: one descriptor read per gate + every site tensor of the final state
    # host-synchronised: two descriptor uploads per gate (run, finalize), one read;
    # resident: one upload per gate, the descriptors read once at the end (statistics)
    h2d = ngates * 16 * 8 + ngates * (1 if RESIDENT else 2) * 32 * 8
    d2h = ngates * 32 * 8 + sum(t.numel() * t.element_size() for t in res) + (4 * (N_QUBITS + 1) if RESIDENT else 0)
    e2e = {"value": ngates * ws / (e2e_ms / 1000.0), "unit": "gates/s", "h2d_bytes_per_step": h2d,
           "d2h_bytes_per_step": d2h}

    # ---------------------------------------------------------------- the other execution mode (same timing)
    alt_ms = 0.0
    alt = None
    for _ in range(args.steps):
        flush_buf.zero_()
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        alt = run_ours(ops_dev, device, resident=not RESIDENT)
        e.record()
        e.synchronize()
        alt_ms += s.elapsed_time(e)
    alt_ms = max_over_ranks(dist, alt_ms, device) / args.steps
    other_mode = {"execution": "host-synchronised (ranks read back after every batch)" if RESIDENT else
                  "device-resident (no host sync between batches)",
                  "value": ngates * ws / (alt_ms / 1000.0), "unit": "gates/s"}

    if rank != 0:
        if dist is not None:
            dist.destroy_process_group()
        return

    # ---------------------------------------------------------------- roofline of the dominant kernel
    hbm, bf16, src = peaks()
    kernels = {k: v for k, v in stage_ms.items() if k != "host_gap"}
    dom = max(kernels, key=kernels.get)
    # algorithmic work of each stage per step (sizes from the step's own statistics:
    # gate on bond q has X of (2 chiL) x (2 chiR) with chiL = bond q-1, chiR = bond q+1)
    work = {}
    bd = last.statistics.logs
    sizes = []
    tl = [1] * (N_QUBITS - 1)
    for (_, q, _), k in zip(ops_host, bd["k_star"]):
        chiL = 1 if q == 0 else tl[q - 1]
        chiR = 1 if q == N_QUBITS - 2 else tl[q + 1]
        sizes.append((2 * chiL, 2 * chiR, k))
        tl[q] = k
    for m_, n_, k in sizes:
        fl_tri = 16.0 / 3.0 * n_ ** 3
        by_tri = 2.0 * n_ * n_ * 8
        work.setdefault("tridiag", [0.0, 0.0])
        work["tridiag"][0] += by_tri
        work["tridiag"][1] += fl_tri
        work.setdefault("gram", [0.0, 0.0])
        work["gram"][0] += (m_ * n_ + n_ * n_) * 8
        work["gram"][1] += 8.0 * m_ * n_ * n_
        work.setdefault("xv", [0.0, 0.0])
        work["xv"][0] += (m_ * n_ + n_ * k + m_ * k) * 8
        work["xv"][1] += 8.0 * m_ * n_ * k
        work.setdefault("backtransform", [0.0, 0.0])
        work["backtransform"][0] += (n_ * n_ + 2 * n_ * k) * 8
        work["backtransform"][1] += 8.0 * n_ * n_ * k
    wb, wf = work.get(dom, [0.0, 0.0])
    t_dom = stage_ms[dom] / 1000.0
    bound = "tensor" if dom in ("gram", "xv") else "hbm"
    if bound == "hbm":
        achieved = wb / t_dom / 1e9 if t_dom > 0 else 0.0
        roof = {"bound": "hbm", "achieved": achieved, "peak": hbm, "unit": "GB/s",
                "frac": achieved / hbm, "traffic": None}
    else:
        achieved = wf / t_dom / 1e12 if t_dom > 0 else 0.0
        roof = {"bound": "tensor", "achieved": achieved, "peak": bf16, "unit": "TFLOP/s",
                "frac": achieved / bf16, "traffic": None}
    roof.update({"kernel": dom, "peak_source": src, "stage_ms_per_step": {k: round(v, 3) for k, v in stage_ms.items()},
                 "algorithmic_flops_per_step": wf, "algorithmic_bytes_per_step": wb})
    if dom == "tridiag":
        # The Householder reduction keeps each matrix in the registers and shared
        # memory of a cluster, so HBM is not what limits it: one launch per layer
        # runs n - 1 dependent column steps, each a pass over the own rows and two
        # exchanges, by one 8-warp CTA per SM (its rows fill the register file).
        # Its FP32 rate is reported beside the HBM fraction of the contract.
        fp32_peak = 152 * 128 * 2 * (clocks.get("sm_max_mhz") or 2070.0) / 1e6  # TFLOP/s, SIMT FMA
        roof["limiter"] = ("latency: n - 1 dependent column steps (pass over the own rows, norm, reflector, two "
                           "exchanges) at ~35% issue activity, one 8-warp CTA per SM (not HBM)")
        roof["fp32_simt"] = {"achieved_tflops": wf / t_dom / 1e12 if t_dom > 0 else 0.0,
                             "peak_tflops": fp32_peak,
                             "frac": (wf / t_dom / 1e12) / fp32_peak if t_dom > 0 else 0.0}
        # DRAM bytes of ONE launch (one saturated layer: 20 Gram matrices of
        # 512 x 512) from an ncu capture of this kernel on 20 matrices of that
        # size: read 21 733 120 B, written 0 B, against that launch's 20 x 2 n^2 x
        # 8 B = 83 886 080 algorithmic bytes (the rest is served from L2, where the
        # Gram GEMM left it).  Per launch, not per step.
        roof["traffic"] = 21733120
        roof["traffic_per_launch"] = {"matrices": 20, "n": 512, "algorithmic_bytes": 20 * 2 * 512 * 512 * 8,
                                      "dram_bytes": 21733120,
                                      "source": "ncu dram__bytes_read.sum + dram__bytes_write.sum, one launch"}

    line = {"metric": METRIC, "value": value, "unit": "gates/s", "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms_per_step, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "complex64", "data": "synthetic",
            "config": config_of(ws),
            "implementation": {
                "l2": "flushed between timed steps (2x L2 write)",
                "precision": "complex64; Gram / X.V / polish GEMMs on tcgen05 (3xTF32), FP32 eigensolver",
                "tridiagonalisation": ("two-stage (band reduction + bulge chasing)" if args.two_stage else
                                       "one-stage, matrix in cluster registers and shared memory"),
                "execution": "device-resident (no host sync between batches)" if RESIDENT else
                             "host-synchronised (ranks read back after every batch)"},
            "clocks": clocks, "gpu_launches": launches, "e2e": e2e, "roofline": roof, "other_mode": other_mode}

    # ---------------------------------------------------------------- CUDA-graph replay of the same circuit
    # MPSBatch.capture records every launch of the circuit once (device-resident,
    # start state restored at the head of the graph); each replay is one launch
    if not args.no_graph:
        cap = aq.MPSBatch([aq.AdaptiveMPS(N_QUBITS, bond_dim=1, eps_bond=EPS, chi_max_per_bond=CHI, device=device,
                                          device_resident=True)]).capture([ops_dev])
        for _ in range(2):
            cap.replay()
        torch.cuda.synchronize()
        g_ms = 0.0
        for _ in range(args.steps):
            flush_buf.zero_()
            torch.cuda.synchronize()
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            s.record(cap.stream)
            cap.replay()
            e.record(cap.stream)
            e.synchronize()
            g_ms += s.elapsed_time(e)
        g_ms /= args.steps
        cap.finish()
        line["graph_replay"] = {"value": ngates / (g_ms / 1000.0), "unit": "gates/s", "ms_per_step": g_ms,
                                "kernels_per_replay": cap.kernels_per_replay,
                                "what": "the same circuit captured once (MPSBatch.capture) and replayed as one "
                                        "CUDA graph: no host enqueue between layers"}

    # ---------------------------------------------------------------- FP64 reference state
    # this package's complex128 run (host-synchronised) of the same circuit
    t0 = time.perf_counter()
    m64 = run_ours(ops_dev, device, dtype=torch.complex128, resident=False)
    torch.cuda.synchronize()
    t64 = time.perf_counter() - t0
    n64 = mps_overlap(m64.tensors, m64.tensors).real

    def fid64(ts, ref=None):
        ref = m64.tensors if ref is None else ref
        f = mps_overlap(ts, ref)
        return abs(f) ** 2 / (mps_overlap(ts, ts).real * mps_overlap(ref, ref).real)

    # the same after the first 150 gates, before the chi cap truncates anything
    # the float32 rank rule can see: there every float32 arm must agree with FP64
    # to 1 - 1e-6; after the cap binds, float32 rounding decides which of two
    # near-equal values is dropped and every float32 run (the reference's own
    # complex64 vs complex128 too) drifts chaotically (0.57-0.83 after 390 gates)
    N_EARLY = 150
    m64e = run_ours(ops_dev[:N_EARLY], device, dtype=torch.complex128, resident=False).tensors
    early = {"ours": fid64(run_ours(ops_dev[:N_EARLY], device).tensors, m64e)}
    line["fidelity_vs_fp64"] = {"value": fid64(last.tensors), "fp64_gpu_seconds": t64,
                                "what": "|<psi|psi_fp64>|^2 of the final state; psi_fp64 = this package's complex128 run",
                                "after_150_gates": early["ours"]}

    # ---------------------------------------------------------------- plain form on the same GPU
    if not args.no_plain:
        plain_gpu_circuit(ops_dev[:60], device)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        pt = plain_gpu_circuit(ops_dev, device)
        torch.cuda.synchronize()
        tp = time.perf_counter() - t0
        f = mps_overlap([t for t in last.tensors], pt)
        fa = mps_overlap(last.tensors, last.tensors).real
        fb = mps_overlap(pt, pt).real
        line["plain_gpu"] = {"value": ngates / tp, "unit": "gates/s",
                             "what": "reference call sequence on this GPU: torch complex64 einsum + torch.linalg.svd (cuSOLVER) + host rank rule",
                             "fidelity_vs_ours": abs(f) ** 2 / (fa * fb), "fidelity_vs_fp64": fid64(pt),
                             "fidelity_vs_fp64_after_150_gates": fid64(plain_gpu_circuit(ops_dev[:N_EARLY], device),
                                                                       m64e)}

    # ---------------------------------------------------------------- learned-rank arm
    from atlasq_gb300 import rank_predictor as rp
    wpath = rp.default_predictor_path("brickwork40")
    if not args.no_learned and os.path.exists(wpath):
        pred = rp.load_predictor(wpath, device=device)

        def run_learned(ops=ops_dev):
            m = aq.AdaptiveMPS(N_QUBITS, bond_dim=1, eps_bond=EPS, chi_max_per_bond=CHI, device=device)
            m.rank_predictor = pred
            for _, q, U in ops:
                m.apply_two_site_gate(q, U)
            m.flush()
            return m
        run_learned()
        lm_ms, ml = 0.0, None
        for _ in range(args.steps):
            flush_buf.zero_()
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            s.record()
            ml = run_learned()
            e.record()
            e.synchronize()
            lm_ms += s.elapsed_time(e)
        lm_ms /= args.steps
        plain_host = alt if RESIDENT else last
        line["learned"] = {
            "value": ngates / (lm_ms / 1000.0), "unit": "gates/s", "fidelity_vs_fp64": fid64(ml.tensors),
            "fidelity_vs_fp64_after_150_gates": fid64(run_learned(ops_dev[:N_EARLY]).tensors, m64e),
            "execution": "host-synchronised; the MLP (agb_mlp_forward) sizes each gate's eigenpair count",
            "predictor": ("5-64-64-64-1 MLP trained on the GPU on plain runs of the 40-qubit brickwork "
                          "(depth 20, chi_max 256; seeds 2000-2015, disjoint from this circuit's)"),
            "rank_fallbacks": ml.rank_fallbacks,
            "eigenpairs_vs_plain_host": ml.ell_total / max(plain_host.ell_total, 1),
            "same_bond_dims_as_plain_host": list(ml.bond_dims) == list(plain_host.bond_dims)}

    # ---------------------------------------------------------------- CPU baseline (oracle port)
    if not args.no_cpu_baseline:
        cap = float(os.environ.get("AGB_CPU_BASELINE_CAP_S", "30"))
        g, t = cpu_port_circuit(ops_host, time_cap=cap)
        line["cpu_baseline"] = {"value": g / t, "unit": "gates/s", "cores": os.cpu_count() or 1, "kind": "port",
                                "sample": (f"first {g} of 390 gates in circuit order (capped at {cap:.0f} s)"
                                           if g < ngates else "full 390-gate circuit") +
                                          PORT_NOTE}
    print(json.dumps(line), flush=True)
    if dist is not None:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
