"""Timed cases: the work that programs using this library have it do, through its public entry points.

Kinds of case (``case["kind"]``):

* ``slot``  - one execution of a slot plan (``PuschSlotPlan.execute_device``, CUDA graph on a stream of the program's own) on
  grids in device memory: DM-RS estimation, demodulation, rate dematching, LDPC, TB assembly, optionally with the learned
  estimator or with UCI on PUSCH.
* ``host``  - one ``pg_pusch_plan_execute_host`` call: grids from pinned host memory, TBs and results back to it.
* ``ldpc``  - one batched LDPC decode (``LdpcBatchDecoder.decode_device``).
* ``harq``  - two transmissions of a list of codeblocks: rate dematching of rv 0, combining of rv 2, LDPC decode.
* ``train`` - one forward and backward pass of the learned estimator's network, gradients read back.

The allocations of a case (cells, UEs, MCS) are fixed by ``case["layout"]``; the transport blocks, channels and noise come from
the seed. Inputs are the project's simulator's: exponential-PDP Rayleigh channels, AWGN, link adaptation as in its benchmark.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ocudu-dapp-platform_b200"))

from pusch_b200 import _native, codec, learned, mcs, sim, uci  # noqa: E402
from pusch_b200._native import PgLdpcCb, PgPuschUci, PgRmCb, PgSchResult  # noqa: E402
from pusch_b200.ldpc import LdpcBatchDecoder, make_descriptors  # noqa: E402
from pusch_b200.pusch import PgPortResult, PuschSlotPlan  # noqa: E402

MAX_ITER = 6


def listed():
    return [
        # A small cell with one scheduled UE: 20 MHz, QPSK, one layer, two receive ports. Latency and launches.
        dict(name="slot_20mhz_single_ue", kind="slot", layout=0, cells=0, max_ues=1, nof_rb=51, mcs_table=1, mcs=5, layers=1, ports=2,
             dmrs=1, snr=10.0, learned=False, uci=False, autotune=False),
        # One UE on a whole 100 MHz carrier at 256QAM, two layers, four receive ports: the peak-rate slot.
        dict(name="slot_100mhz_full_cell", kind="slot", layout=0, cells=0, max_ues=1, nof_rb=273, mcs_table=2, mcs=20, layers=2, ports=4,
             dmrs=2, snr=25.0, learned=False, uci=False, autotune=False),
        # Three cells of a site with up to 16 UEs each, launch shapes as the plan has them.
        dict(name="slot_3_cells", kind="slot", layout=3, cells=3, max_ues=16, learned=False, uci=False, autotune=False),
        # The benchmark's batched uneven slot: 16 cells of 1 to 16 UEs, QPSK to 256QAM, tuned as a program that keeps a plan tunes it.
        dict(name="slot_16_cells", kind="slot", layout=0, cells=16, max_ues=16, learned=False, uci=False, autotune=True),
        # The same with the learned estimator refining the UEs at 64QAM and above (the benchmark's headline).
        dict(name="slot_16_cells_learned", kind="slot", layout=0, cells=16, max_ues=16, learned=True, uci=False, autotune=True),
        # Four cells whose UEs carry HARQ-ACK and CSI Part 1 on PUSCH: short-block and polar-coded messages.
        dict(name="slot_4_cells_uci", kind="slot", layout=5, cells=4, max_ues=16, learned=False, uci=True, autotune=False),
        # A slot that arrives in host memory and whose TBs go back there, one call at a time.
        dict(name="host_6_cells", kind="host", layout=2, cells=6, max_ues=16, learned=False, uci=False, autotune=False),
        # The codeblocks of one mid-size transport block handed to the batch decoder: latency.
        dict(name="ldpc_6_codeblocks", kind="ldpc", n=6, z=384, bg_mix=1.0, ebn0_min=1.5, ebn0_max=3.0, max_iterations=10),
        # The decoder batch of the benchmark: 512 codeblocks of both base graphs at the largest lifting size.
        dict(name="ldpc_512_codeblocks", kind="ldpc", n=512, z=384, bg_mix=0.5, ebn0_min=1.0, ebn0_max=3.0, max_iterations=10),
        # Codeblocks of many sizes (odd lifting sizes, fillers, every modulation) in their second transmission.
        dict(name="harq_200_codeblocks", kind="harq", layout=1, groups=25, per_group=8, max_iterations=6),
        # One training pass of the learned estimator at the training script's batch size.
        dict(name="train_96k_rows", kind="train", layout=0, rows=96000),
    ]


def draw(rng):
    kind = rng.choice(["single", "single", "slot", "slot", "slot", "host", "ldpc", "ldpc", "harq", "train"])
    layout = rng.randrange(1 << 20)
    if kind == "single":
        layers = rng.choice([1, 2])
        ports = rng.choice([p for p in (1, 2, 4) if p >= layers])
        table = rng.choice([1, 2])
        index = rng.randrange(len(mcs.MCS_TABLE_1 if table == 1 else mcs.MCS_TABLE_2))
        qm, r = mcs.mcs(table, index)
        return dict(kind="slot", layout=layout, cells=0, max_ues=1, nof_rb=_log_int(rng, 2, 273), mcs_table=table, mcs=index,
                    layers=layers, ports=ports, dmrs=rng.choice([1, 2]),
                    snr=float(sim.required_snr_db(qm, r, layers, ports)) + rng.uniform(1.0, 4.0), learned=False, uci=False,
                    autotune=False)
    if kind in ("slot", "host"):
        return dict(kind=kind, layout=layout, cells=_log_int(rng, 1, 16 if kind == "slot" else 6), max_ues=rng.randint(1, 16),
                    learned=kind == "slot" and rng.random() < 0.4, uci=kind == "slot" and rng.random() < 0.3,
                    autotune=kind == "slot" and rng.random() < 0.3)
    if kind == "ldpc":
        z = rng.choice([z for z in codec.LIFTING_SIZES if z >= 16] + [384] * 12)
        return dict(kind="ldpc", n=_log_int(rng, 1, 512), z=z, bg_mix=rng.choice([0.0, 0.3, 0.5, 1.0]),
                    ebn0_min=1.0 + rng.random(), ebn0_max=3.0 + rng.random(),
                    max_iterations=rng.choice([6, 8, 10]))
    if kind == "harq":
        return dict(kind="harq", layout=layout, groups=_log_int(rng, 2, 25), per_group=rng.randint(1, 8), max_iterations=6)
    return dict(kind="train", layout=layout, rows=_log_int(rng, 2000, 96000))


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# ---------------------------------------------------------------------------------------------------------------------
# What the program keeps for its lifetime: one context and one stream.

@functools.lru_cache(maxsize=None)
def _context():
    return _native.Context(device=0, max_codeblocks=1024)


@functools.lru_cache(maxsize=None)
def _stream():
    return torch.cuda.Stream()


# ---------------------------------------------------------------------------------------------------------------------
# Slots.

def _cells(case):
    """Per cell (UE list, receive ports, carrier PRBs): one UE, or the simulator's uneven cells (1 to max_ues UEs on contiguous
    allocations of a 273-PRB carrier, SNR U[0, 30] dB, MCS among those the SNR supports)."""
    if case["cells"] == 0:
        ue = sim.ue_from_mcs(0, case["nof_rb"], case["layers"], case["mcs_table"], case["mcs"], (2, 11)[:case["dmrs"]],
                             snr_db=case["snr"], channel="pdp" if case["nof_rb"] > 100 else "flat")
        return [([ue], case["ports"], case["nof_rb"])]
    rng = np.random.default_rng(case["layout"])
    out = []
    for cell in range(case["cells"]):
        n = int(rng.integers(1, case["max_ues"] + 1))
        used = int(rng.integers(200, 274))
        cuts = np.sort(rng.choice(np.arange(1, used), size=n - 1, replace=False)) if n > 1 else []
        edges = [0, *[int(c) for c in cuts], used]
        ues = []
        for u in range(n):
            layers, snr = int(rng.integers(1, 3)), float(rng.uniform(0.0, 30.0))
            ok = []
            for layers in ([2, 1] if layers == 2 else [1]):
                ok = [i for i, (qm, r) in enumerate(mcs.MCS_TABLE_2) if sim.required_snr_db(qm, r, layers, 4) <= snr]
                if ok:
                    break
            top = max(ok) if ok else 0
            index = int(rng.integers(max(0, top - 3), top + 1))
            ues.append(sim.ue_from_mcs(edges[u], edges[u + 1] - edges[u], layers, 2, index, (2, 11), snr_db=snr, channel="pdp",
                                       rnti=0x4000 + 16 * cell + u, n_id=cell, n_id_data=cell))
        out.append((ues, 4, 273))
    return out


def _slots(case, seed):
    """The received slots. With UCI the transport blocks (and UCI messages) are all zeros, whose coded bits are zeros in every
    stream wherever the multiplexer puts them; the scrambled symbols are as random as any."""
    rng = np.random.default_rng([case["layout"], seed])
    out = []
    for c, (ues, ports, prb) in enumerate(_cells(case)):
        tb = [np.zeros(ue.tbs_bits, np.uint8) for ue in ues] if case["uci"] else None
        out.append(sim.make_pusch_slot(ues, ports, nof_prb_grid=prb, slot=c % 20, seed=int(rng.integers(0, 2 ** 31)), tb_bits=tb))
    return out


def _uci_of(case, ues):
    """HARQ-ACK of 3 to 11 bits on every larger allocation, CSI Part 1 of 4 to 60 bits on two of three; the encoded sizes from
    the grant. All-zero entries carry none."""
    rng = np.random.default_rng([case["layout"], 77])
    out = []
    for ue in ues:
        q = PgPuschUci()
        ack, csi = int(rng.choice([3, 4, 5, 8, 11])), int(rng.choice([0, 4, 8, 11, 24, 60]))
        if ue.nof_rb >= 8:
            s = uci.ulsch_information(ue.tbs_bits, ue.base_graph, ue.modulation_order, ue.nof_layers, ue.nof_rb, 0, 14,
                                      sum(1 << d for d in ue.dmrs_symbols), nof_harq_ack_bits=ack, nof_csi_part1_bits=csi)
            if csi > 11 and s["nof_csi_part1_bits"] < 2 * csi + 40:
                csi = 0
                s = uci.ulsch_information(ue.tbs_bits, ue.base_graph, ue.modulation_order, ue.nof_layers, ue.nof_rb, 0, 14,
                                          sum(1 << d for d in ue.dmrs_symbols), nof_harq_ack_bits=ack)
            q.nof_harq_ack_bits, q.nof_csi_part1_bits, q.nof_cdm_groups_without_data = ack, csi, 2
            q.nof_enc_harq_ack_bits, q.nof_enc_csi_part1_bits = s["nof_harq_ack_bits"], s["nof_csi_part1_bits"]
            q.nof_harq_ack_rvd = s["nof_harq_ack_rvd"]
        out.append(q)
    return out


class _Slot:
    pass


def _prepare_slot(case, seed):
    s = _Slot()
    ctx = _context()
    slots = _slots(case, seed)
    ues = [ue for sl in slots for ue in sl.ues]
    s.uci = _uci_of(case, ues) if case["uci"] else None
    s.plan = PuschSlotPlan(ctx, slots, max_iterations=MAX_ITER, graph=True, uci=s.uci)
    n = s.plan.n
    s.grid = torch.from_numpy(s.plan.grid.view(np.int32)).cuda()
    s.tb = torch.zeros(max(1, s.plan.tb_bytes), dtype=torch.uint8, device="cuda")
    s.res = torch.zeros(n * ctypes.sizeof(PgSchResult), dtype=torch.uint8, device="cuda")
    s.ports = torch.zeros((n * 4, 5), dtype=torch.float32, device="cuda")
    if case["learned"]:
        use = [ue.modulation_order >= 6 for ue in ues]
        if any(use):
            s.net = learned.LearnedEstimator(ctx, s.plan.le_rows(use), params=learned.load_params())
            s.plan.set_learned(s.net, use)
    if case["autotune"]:
        torch.cuda.synchronize()
        s.plan.autotune(s.grid.data_ptr(), reps=5)
    s.polar = [(u, k, b) for u, q in enumerate(s.uci or []) for k, b in ((0, q.nof_harq_ack_bits), (1, q.nof_csi_part1_bits)) if b > 11]
    torch.cuda.synchronize()
    return s


def _run_slot(s):
    st = _stream()
    s.plan.execute_device(s.grid.data_ptr(), s.tb.data_ptr(), s.res.data_ptr(), s.ports.data_ptr(), st.cuda_stream)
    out = {"tb": s.tb, "results": s.res, "ports": s.ports}
    if s.uci is not None:
        st.synchronize()  # the UCI results are read from the plan once its execution has completed
        out["uci"] = np.frombuffer(s.plan.uci_results(), np.uint8).copy()
        msgs = [s.plan.uci_message(u, k, b) for u, k, b in s.polar]
        out["uci_polar"] = np.concatenate([np.append(b, np.uint8(v)) for b, v in msgs]) if msgs else np.zeros(1, np.uint8)
    return out


def _prepare_host(case, seed):
    s = _Slot()
    s.plan = PuschSlotPlan(_context(), _slots(case, seed), max_iterations=MAX_ITER, graph=True)
    n = s.plan.n
    s.grid = torch.from_numpy(s.plan.grid.view(np.int32)).pin_memory()
    s.tb = torch.zeros(max(1, s.plan.tb_bytes), dtype=torch.uint8).pin_memory()
    s.res = torch.zeros(n * ctypes.sizeof(PgSchResult), dtype=torch.uint8)
    s.ports = torch.zeros((n * 4, 5), dtype=torch.float32)
    s.used = np.repeat([d.nof_rx_ports for d in s.plan.descs], 4).reshape(n, 4) > np.arange(4)
    assert ctypes.sizeof(PgPortResult) == 20
    return s


def _run_host(s):
    p = s.plan
    p.ctx.check(p.lib.pg_pusch_plan_execute_host(p.handle, s.grid.data_ptr(), s.tb.data_ptr(), p.tb_bytes, s.res.data_ptr(),
                                                 s.ports.data_ptr()))
    return {"tb": s.tb, "results": s.res, "ports": s.ports.reshape(-1, 4, 5)[torch.from_numpy(s.used)]}


def _work_slot(case):
    """Bytes: the occupied grid words once, TBs and results once. Operations: the learned network's, and one LDPC iteration of
    every codeblock (10 integer operations per edge and lifted lane over the check rows its bits reach)."""
    cells = _cells(case)
    nbytes, ops = 0, 0
    for ues, ports, _ in cells:
        for ue in ues:
            nbytes += ports * 14 * 12 * ue.nof_rb * 4 + ue.tbs_bits // 8 + ctypes.sizeof(PgSchResult) + 20 * ports
            if case["learned"] and ue.modulation_order >= 6:
                ops += 512000 * ports * ue.nof_layers * 12 * ue.nof_rb
            ncs = sim.nof_ch_symbols(ue)
            seg = codec.segment_tx(ue.tbs_bits, ue.base_graph, ue.modulation_order, ue.nof_layers, ncs)
            ops += seg["nof_cbs"] * _ldpc_ops(ue.base_graph, seg["lifting_size"], seg["e_long"] + seg["nof_filler_bits"])
    return {"bytes": nbytes, "flops": ops}


def _ldpc_ops(bg, z, filled):
    kb, rows = (22, 46) if bg == 1 else (10, 42)
    n = min(rows, max(4, -(-(filled + 2 * z) // z) - kb))
    return 10 * int(codec.base_graph(bg)[0][:n].sum()) * z


# ---------------------------------------------------------------------------------------------------------------------
# LDPC batches.

def _prepare_ldpc(case, seed):
    s = _Slot()
    bgs = np.where(np.random.default_rng(case["n"]).permutation(case["n"]) < round(case["bg_mix"] * case["n"]), 1, 2).astype(np.int32)
    batch = sim.ldpc_batch(seed=seed, n=case["n"], z=case["z"], ebn0_range=(case["ebn0_min"], case["ebn0_max"]), bgs=bgs,
                           max_iterations=case["max_iterations"])
    s.n = case["n"]
    s.descs, llrs, nbits = make_descriptors(batch.jobs)
    s.dec = LdpcBatchDecoder(context=_context())
    s.llrs = torch.from_numpy(llrs).cuda()
    s.bits = torch.zeros(nbits, dtype=torch.uint8, device="cuda")
    s.iters = torch.zeros(s.n, dtype=torch.int32, device="cuda")
    return s


def _run_ldpc(s):
    s.dec.decode_device(s.descs, s.n, s.llrs.data_ptr(), s.bits.data_ptr(), s.iters.data_ptr(), _stream().cuda_stream)
    return {"bits": s.bits, "iterations": s.iters}


def _work_ldpc(case):
    """About five iterations at these Eb/N0; the share of base graph 1 is case["bg_mix"]."""
    n, z, f = case["n"], case["z"], case["bg_mix"]
    per = f * _ldpc_ops(1, z, 66 * z) + (1 - f) * _ldpc_ops(2, z, 50 * z)
    return {"bytes": int(n * (f * (66 + 22 / 8) + (1 - f) * (50 + 10 / 8)) * z) + 24 * n, "flops": int(5 * n * per)}


# ---------------------------------------------------------------------------------------------------------------------
# Codeblocks in their second transmission.

def _groups(case):
    """Groups of equal codeblocks, as the transport blocks of a slot have: (base graph, Z, Qm, fillers, E of each transmission)."""
    rng = np.random.default_rng([case["layout"], 3])
    sizes = [z for z in codec.LIFTING_SIZES if z >= 10]
    out = []
    for _ in range(case["groups"]):
        bg, qm = int(rng.integers(1, 3)), int(rng.choice([2, 4, 6, 8]))
        z = int(sizes[-1 - min(len(sizes) - 1, int(rng.exponential(9.0)))])
        k = (22 if bg == 1 else 10) * z
        fill = int(rng.integers(0, 2 * z)) // 8 * 8
        rate = rng.uniform(0.45, 0.93) if bg == 1 else rng.uniform(0.25, 0.67)
        out.append((bg, z, qm, fill, int((k - fill) / rate) // qm * qm))
    return out


def _prepare_harq(case, seed):
    rng = np.random.default_rng([case["layout"], seed])
    jobs = []
    for bg, z, qm, fill, e in _groups(case):
        k = (22 if bg == 1 else 10) * z
        poly = 2 if case["per_group"] > 1 else 1
        msg = codec.attach_crc(poly, rng.integers(0, 2, (case["per_group"], k - fill - 24), dtype=np.uint8))
        cw = codec.ldpc_encode(bg, z, np.concatenate([msg, np.zeros((case["per_group"], fill), np.uint8)], axis=1))
        # About 2 dB short of what one transmission needs.
        sigma2 = 1.0 / (2.0 ** (2.0 * (k - fill) / e) - 1.0) * 10 ** (0.1 * rng.uniform(0.0, 2.0))
        llr = []
        for rv in (0, 2):
            x = 1.0 - 2.0 * codec.rate_match(bg, z, cw, e, rv=rv, qm=qm, nof_filler_bits=fill)
            y = x + math.sqrt(sigma2) * rng.standard_normal(x.shape)
            llr.append(np.clip(np.rint(8.0 * y / sigma2), -120, 120).astype(np.int8))
        jobs += [(bg, z, qm, fill, e, poly, llr[0][i], llr[1][i]) for i in range(case["per_group"])]
    s = _Slot()
    s.n = len(jobs)
    s.first, s.second, s.cbs = (PgRmCb * s.n)(), (PgRmCb * s.n)(), (PgLdpcCb * s.n)()
    io, oo, bo = 0, 0, 0
    for i, (bg, z, qm, fill, e, poly, _, _) in enumerate(jobs):
        n = (66 if bg == 1 else 50) * z
        for d, rv, new in ((s.first[i], 0, 1), (s.second[i], 2, 0)):
            d.in_offset, d.rm_length, d.out_offset, d.nref = io, e, oo, 0
            d.lifting_size, d.nof_filler_bits, d.base_graph, d.rv, d.modulation_order, d.new_data = z, fill, bg, rv, qm, new
        c = s.cbs[i]
        c.llr_offset, c.nof_llrs, c.out_offset, c.lifting_size, c.nof_filler_bits = oo, n, bo, z, fill
        c.base_graph, c.crc_poly, c.max_iterations = bg, poly, case["max_iterations"]
        io, oo, bo = io + e, oo + (n + 15) // 16 * 16, bo + (n // (66 if bg == 1 else 50) * (22 if bg == 1 else 10) + 7) // 8
    s.rx = [torch.from_numpy(np.concatenate([j[k] for j in jobs])).cuda() for k in (6, 7)]
    s.soft = torch.zeros(oo, dtype=torch.int8, device="cuda")
    s.bits = torch.zeros(bo, dtype=torch.uint8, device="cuda")
    s.iters = torch.zeros(s.n, dtype=torch.int32, device="cuda")
    s.dec = LdpcBatchDecoder(context=_context())
    return s


def _run_harq(s):
    ctx, st = s.dec.ctx, _stream().cuda_stream
    for d, x in ((s.first, s.rx[0]), (s.second, s.rx[1])):
        ctx.check(ctx.lib.pg_rate_dematch_batch_device(ctx.handle, ctypes.addressof(d), s.n, x.data_ptr(), s.soft.data_ptr(), st))
    s.dec.decode_device(s.cbs, s.n, s.soft.data_ptr(), s.bits.data_ptr(), s.iters.data_ptr(), st)
    return {"soft": s.soft, "bits": s.bits, "iterations": s.iters}


def _work_harq(case):
    nbytes, ops = 0, 0
    for bg, z, _, fill, e in _groups(case):
        n, k = (66 if bg == 1 else 50) * z, (22 if bg == 1 else 10) * z
        nbytes += case["per_group"] * (2 * e + n + k // 8)
        ops += 2 * case["per_group"] * _ldpc_ops(bg, z, n)  # rv 2 reaches the last check rows; about two iterations
    return {"bytes": nbytes, "flops": ops}


# ---------------------------------------------------------------------------------------------------------------------
# Training pass of the learned estimator.

def _train_inputs(case, seed):
    """Rows of allocations of 1 to 273 PRBs with two zero rows before each, features and output gradients as bf16 values."""
    rng = np.random.default_rng([case["layout"], 9])
    rows = case["rows"]
    valid = np.zeros(rows, np.uint8)
    r = 2
    while r < rows:
        n = min(rows - r, 12 * int(round(math.exp(rng.uniform(0.0, math.log(273))))))
        valid[r:r + n] = 1
        r += n + 2
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + case["layout"])
    v = torch.from_numpy(valid).cuda()
    x = (0.7 * torch.randn((rows, 16), generator=g, device="cuda") * v[:, None]).bfloat16()
    dy = (torch.randn((rows, 16), generator=g, device="cuda") * v[:, None] / rows).bfloat16()
    return x, dy, v


def _chunked(a):
    """[rows][16] -> the library's activation layout [2][rows][8]."""
    return a.reshape(a.shape[0], 2, 8).permute(1, 0, 2).contiguous()


def _prepare_train(case, seed):
    s = _Slot()
    x, dy, s.valid = _train_inputs(case, seed)
    s.rows = case["rows"]
    s.x, s.dy = _chunked(x), _chunked(dy)
    s.y = torch.zeros((2, s.rows, 8), dtype=torch.bfloat16, device="cuda")
    s.net = learned.LearnedEstimator(_context(), s.rows, params=learned.load_params())
    return s


def _run_train(s):
    st = _stream().cuda_stream
    s.net.forward(s.x.data_ptr(), s.valid.data_ptr(), s.rows, s.y.data_ptr(), st)
    s.net.backward(s.dy.data_ptr(), s.rows, st)
    return {"y": s.y, "grads": s.net.grads()}


def _work_train(case):
    return {"bytes": case["rows"] * (32 + 32 + 32 + 1) + 8 * learned.nof_params(), "flops": 3 * 512000 * case["rows"]}


def _exact_train(case, seed):
    """The network and its gradients in float64: 14 convolutions of kernel 5 as matrix products over shifted rows."""
    x, dy, v = _train_inputs(case, seed)
    p = torch.from_numpy(learned.load_params()).cuda().double()
    m = v.double()[:, None]
    layers, o = [], 0
    for cin, cout in [(16, 64)] + [(64, 64)] * 12 + [(64, 16)]:
        layers.append((p[o:o + 5 * cin * cout].reshape(5, cin, cout), p[o + 5 * cin * cout:o + 5 * cin * cout + cout]))
        o += 5 * cin * cout + cout

    def shift(a, t):  # a[r + t], zero outside
        b = torch.zeros_like(a)
        if t >= 0:
            b[:a.shape[0] - t] = a[t:]
        else:
            b[-t:] = a[:t]
        return b

    def conv(a, w, b):
        return sum(shift(a, t - 2) @ w[t] for t in range(5)) + b

    acts, outs, a, skip = [], [], x.double(), None
    for i, (w, b) in enumerate(layers):
        acts.append(a)
        z = conv(a, w, b)
        if 0 < i < 13 and i % 2 == 0:
            z = z + skip
        a = z * m if i == 13 else torch.relu(z) * m
        if i % 2 == 0:
            skip = a
        outs.append(a)
    y = a
    grads, g, res = [None] * 14, dy.double(), None
    for i in reversed(range(14)):
        w, _ = layers[i]
        if i < 13:
            if i % 2 == 0 and res is not None and i < 12:
                g = g + res
            g = g * (outs[i] > 0) * m
            if 0 < i and i % 2 == 0:
                res = g
        dw = torch.stack([shift(acts[i], t - 2).T @ g for t in range(5)])
        grads[i] = torch.cat([dw.reshape(-1), g.sum(0)])
        g = sum(shift(g, 2 - t) @ w[t].T for t in range(5))
    return {"y": _chunked(y).cpu(), "grads": torch.cat(grads).cpu()}


# ---------------------------------------------------------------------------------------------------------------------
# The port results in 64 bits: DM-RS type 1 least squares, raised-cosine smoothing over pilots extended by line fits of magnitude
# and phase, and the noise, RSRP, EPRE and SNR sums of the estimator.

def _gold(c_init, first, n):
    total = 1600 + first + n + 31
    x1, x2 = np.zeros(total, np.uint8), np.zeros(total, np.uint8)
    x1[0] = 1
    x2[:31] = (c_init >> np.arange(31)) & 1
    have, step = 31, 1
    while have < total:
        while 31 * step * 2 <= have:  # the recurrences also hold with every lag times a power of two
            step *= 2
        k = min(28 * step, total - have)
        i = have - 31 * step
        x1[have:have + k] = x1[i + 3 * step:i + 3 * step + k] ^ x1[i:i + k]
        x2[have:have + k] = x2[i + 3 * step:i + 3 * step + k] ^ x2[i + 2 * step:i + 2 * step + k] ^ x2[i + step:i + step + k] ^ x2[i:i + k]
        have += k
    return (x1 ^ x2)[1600 + first:1600 + first + n]


def _taps(nof_rb):
    t = (np.arange(31) - 15) / 10.0
    h = np.sinc(t) * np.cos(np.pi * 0.2 * t) / (1 - (0.4 * t) ** 2)
    half = (min(nof_rb, 3) * 10 + 1) // 2 // 2
    h = h[15 - 2 * half:15 + 2 * half + 1:2]
    return h / h.sum()


def _beyond(p, before):
    n = p.size
    i = np.arange(n, dtype=np.float64)
    mag, ph = np.polyfit(i, np.abs(p), 1), np.polyfit(i, np.unwrap(np.angle(p)), 1)
    at = i + (-n if before else n)
    rho = np.polyval(mag, at)
    return np.abs(rho) * np.exp(1j * (np.polyval(ph, at) + np.where(rho > 0, 0, np.pi)))


def _exact_ports(case, seed):
    out = []
    for sl in _slots(case, seed):
        g = sl.grid
        g = (g << 16).view(np.float32).astype(np.float64) + 1j * (g & np.uint32(0xFFFF0000)).view(np.float32).astype(np.float64)
        beta = float(np.float32(10 ** (3 / 20)))
        for ue in sl.ues:
            npil, nd, nl = 6 * ue.nof_rb, len(ue.dmrs_symbols), ue.nof_layers
            pil = []
            for s in ue.dmrs_symbols:
                c = _gold(((14 * sl.slot + s + 1) * (2 * ue.n_id + 1) * (1 << 17) + 2 * ue.n_id) % (1 << 31), 12 * ue.rb_start, 2 * npil)
                r = ((1.0 - 2.0 * c[0::2]) + 1j * (1.0 - 2.0 * c[1::2])) / math.sqrt(2.0)
                pil.append([r * (1.0 - 2.0 * (np.arange(npil) % 2)) if l else r for l in range(nl)])
            pil = np.array(pil)
            taps = _taps(ue.nof_rb)
            nv = npil if ue.nof_rb == 1 else taps.size // 2
            rows = np.zeros((4, 5))
            for p in range(sl.nof_ports):
                rx = g[p, list(ue.dmrs_symbols), 12 * ue.rb_start:12 * (ue.rb_start + ue.nof_rb):2]
                ls = rx[:, None, :] * np.conj(pil)
                if nl > 1:
                    ls = np.repeat((ls[..., 0::2] + ls[..., 1::2]) / 2, 2, axis=-1)
                ls = ls / beta
                sm = np.zeros_like(ls)
                for d in range(nd):
                    for l in range(nl):
                        e = np.concatenate([_beyond(ls[d, l, :nv], True), ls[d, l], _beyond(ls[d, l, -nv:], False)])
                        sm[d, l] = np.convolve(e, taps, mode="same")[nv:nv + npil]
                rsrp = (np.abs(sm) ** 2).sum(axis=(0, 2)) * beta ** 2 / (npil * nd)
                pred = ((sm.sum(0) * beta / nd)[None] * pil).sum(1)
                noise = max(rsrp.mean() / 1e10, (np.abs(pred - rx) ** 2).sum() / (npil * nd - 1))
                rows[p, 0], rows[p, 1], rows[p, 2] = noise, (np.abs(rx) ** 2).sum() / (npil * nd), rsrp.mean() * nl / beta ** 2 / noise
                rows[p, 3:3 + nl] = rsrp
            out.append(rows if case["kind"] == "slot" else rows[:sl.nof_ports])
    return torch.from_numpy(np.concatenate(out))


# ---------------------------------------------------------------------------------------------------------------------

_PREPARE = {"slot": _prepare_slot, "host": _prepare_host, "ldpc": _prepare_ldpc, "harq": _prepare_harq, "train": _prepare_train}
_RUN = {"slot": _run_slot, "host": _run_host, "ldpc": _run_ldpc, "harq": _run_harq, "train": _run_train}
_WORK = {"slot": _work_slot, "host": _work_slot, "ldpc": _work_ldpc, "harq": _work_harq, "train": _work_train}


def prepare(case, seed):
    s = _PREPARE[case["kind"]](case, seed)
    s.run = _RUN[case["kind"]]
    torch.cuda.synchronize()
    return s


def run(state):
    return state.run(state)


def work(case):
    return _WORK[case["kind"]](case)


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] not in ("slot", "host"):
        return None
    out = {"tb": None, "results": None, "ports": _exact_ports(case, seed)}
    if case["uci"]:
        out["uci"] = out["uci_polar"] = None
    return out
