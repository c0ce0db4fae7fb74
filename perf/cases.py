"""Cases by which the speed of the framework is measured: what its users run, through its public entry points.

Three kinds of call, over the ranges that the workloads, tests and benchmark of this repository span:

  net     one network on the plain path (gsbn_b200.capi.Net): training and recall segments of a stimulus schedule, or a
          host loop of single ticks with spikes read back each tick; ProcUpdLazy or ProcUpdMulti updates;
  batch   many independent networks advanced together (gsbn_b200.batch.BatchEngine);
  recall  noise replicates of one trained network (gsbn_b200.recall.Recall), BF16 or FP32 contraction.

listed() names the cases, draw() gives more of the same ranges, prepare()/run() set one up and make one pass, work()
counts what a pass cannot do without and exact() restates a pass in 64 bits where that has a meaning.
"""
import math
import types

import numpy as np
import torch

from gsbn_b200 import batch, capi, recall

F32 = np.float32
DT, EPS, LGBIAS = 0.001, 1e-4, 9.21
NO_INPUT = 0x7FFFFFFF
CUE = 0.3            # share of the HCUs that a recall cue drives
KEPSC = 0.1          # dt / tau_z of the recall engine's projection
MAX_CELLS = 2.5e7    # of one drawn network
SPIKE_RATE = 0.1     # spikes per HCU and tick: maxfq * dt


# ------------------------------------------------------------------------------------------------ the cases

def listed():
    return [
        # a closed loop on the host (an agent, or the engine's per-tick mode): every tick sets its own input row and
        # reads the spikes back, on the two-population network; the smallest calls there are
        dict(name="online_5x10_10x10", kind="net", variant="lazy", H0=5, H=10, M=10, slots=25, slots1=10, patterns=4,
             train=0, recall=0, ticks=64, hz=10.0),
        # one learning trial of the small fully recurrent network: some patterns with short segments, then their recall
        dict(name="trial_10x10", kind="net", variant="lazy", H0=0, H=10, M=10, slots=100, slots1=0, patterns=3,
             train=100, recall=100, ticks=0, hz=0.0),
        # the two-population network with Poisson input noise: its segments of 80 and 20 ticks
        dict(name="schedule_5x10_10x10", kind="net", variant="lazy", H0=5, H=10, M=10, slots=25, slots1=10,
             patterns=20, train=80, recall=20, ticks=0, hz=10.0),
        # the 100x100 network at density 0.1 (1e7 cells): training, recall, and the learned weights read back
        dict(name="schedule_100x100", kind="net", variant="lazy", H0=0, H=100, M=100, slots=1000, slots1=0,
             patterns=20, train=100, recall=100, ticks=0, hz=0.0),
        # the same with ProcUpdMulti updates (row-only, replaying a spike ring)
        dict(name="multi_100x100", kind="net", variant="multi", H0=0, H=100, M=100, slots=1000, slots1=0,
             patterns=20, train=100, recall=100, ticks=0, hz=0.0),
        # a network of more HCUs than the GPU has SMs
        dict(name="schedule_256x50", kind="net", variant="lazy", H0=0, H=256, M=50, slots=1000, slots1=0,
             patterns=10, train=100, recall=100, ticks=0, hz=0.0),
        # the batch workload: networks of 8-64 HCUs x 5-50 MCUs, each fully recurrent, trained and then recalled
        dict(name="batch_128", kind="batch", members=128, hcu_lo=8, hcu_hi=64, mcu_lo=5, mcu_hi=50, patterns=2,
             train=100, recall=50),
        # the replicate recall workload, both forms of the contraction: 64x64, 4096 replicates, 25% cue, 20 Hz noise
        dict(name="recall_bf16_64x64_4096", kind="recall", form="bf16", H=64, M=64, R=4096, ticks=200, hz=20.0),
        dict(name="recall_fp32_64x64_4096", kind="recall", form="fp32", H=64, M=64, R=4096, ticks=20, hz=20.0),
        # a small network with few replicates, where launches count; its whole state is read back
        dict(name="recall_bf16_16x16_128", kind="recall", form="bf16", H=16, M=16, R=128, ticks=20, hz=20.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["net", "net", "net", "net", "batch", "recall", "recall", "recall"])
    if kind == "net":
        while True:
            H, M = _log(rng, 5, 320), _log(rng, 5, 128)
            slots = _log(rng, min(20, H * M), min(3200, H * M))
            H0 = _log(rng, 3, 12) if H <= 40 and rng.random() < 0.3 else 0
            slots1 = _log(rng, 5, min(400, H * M)) if H0 else 0
            online = rng.random() < 0.2
            train = 0 if online else _log(rng, 20, 120)
            c = dict(kind="net", variant=rng.choice(["lazy", "lazy", "lazy", "multi"]), H0=H0, H=H, M=M, slots=slots,
                     slots1=slots1, patterns=4 if online else min(20, 2000 // train), train=train,
                     recall=0 if online else _log(rng, 20, 100), ticks=_log(rng, 16, 64) if online else 0,
                     hz=rng.choice([0.0, 0.0, 10.0, 20.0]))
            if H * M * slots <= MAX_CELLS and _work_net(c)["bytes"] < 1e10:
                return c
    if kind == "batch":
        hi, mhi = _log(rng, 12, 64), _log(rng, 8, 50)
        return dict(kind="batch", members=_log(rng, 4, 128), hcu_lo=rng.randint(4, hi), hcu_hi=hi,
                    mcu_lo=rng.randint(4, mhi), mcu_hi=mhi, patterns=2, train=_log(rng, 20, 100),
                    recall=_log(rng, 20, 50))
    M = rng.choice([16, 32, 64])
    while True:
        H = 256 // M * _log(rng, 1, 16)
        R = 128 * _log(rng, 1, 32)
        form = rng.choice(["bf16", "fp32"])
        if H * M * R <= (1 << 24) and H * M <= 4096:
            break
    return dict(kind="recall", form=form, H=H, M=M, R=R, ticks=_log(rng, 5, 100 if form == "bf16" else 20),
                hz=rng.choice([0.0, 10.0, 20.0, 40.0]))


# ------------------------------------------------------------------------------------------------ one network

def _pop(H, M):
    return dict(hcu_num=H, mcu_num=M, taum=F32(0.005), wtagain=1.0, maxfq=100.0, igain=1.0, wgain=1.0,
                lgbias=F32(LGBIAS), snoise=0.0)


def _proj(src, dest, slots):
    return dict(src_pop=src, dest_pop=dest, tauzi=F32(0.01), tauzj=F32(0.01), taue=F32(0.02), taup=1.0, maxfq=100.0,
                bgain=1.0, wgain=1.0, tauepsc=0.0, slot_num=float(slots))


def _conn(rng, H, slots, Hs, Ms):
    """each destination HCU is fed by whole source HCUs drawn at random, as many as its slots hold, the last in part"""
    rows = []
    for _ in range(H):
        hcus = np.sort(rng.choice(Hs, size=min(Hs, -(-slots // Ms)), replace=False))
        rows.append((hcus[:, None] * Ms + np.arange(Ms)).reshape(-1)[:slots])
    return np.concatenate(rows).astype(np.int32)


def _rows(rng, patterns, shapes):
    """pattern rows, then their cue rows, and the masks of training and of recall"""
    pats = np.concatenate([rng.integers(0, M, (patterns, H)) for H, M in shapes], axis=1).astype(np.int32)
    n_cued = int(np.ceil(pats.shape[1] * CUE))
    cues = np.where(np.arange(pats.shape[1]) < n_cued, pats, NO_INPUT).astype(np.int32)
    masks = np.stack([np.zeros(pats.shape[1]), np.arange(pats.shape[1]) >= n_cued]).astype(np.float32)
    return np.concatenate([pats, cues]), masks


def _pinned(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True).numpy()


def _prepare_net(c, seed):
    rng = np.random.default_rng(seed)
    shapes = ([(c["H0"], c["M"])] if c["H0"] else []) + [(c["H"], c["M"])]
    pops = [_pop(H, M) for H, M in shapes]
    main = len(pops) - 1
    projs, tables = [], []
    if c["H0"]:
        n0 = min(c["slots"], c["H0"] * c["M"])
        projs.append(_proj(0, 1, n0))
        tables.append(_conn(rng, c["H"], n0, c["H0"], c["M"]))
    own = min(c["slots1"] if c["H0"] else c["slots"], c["H"] * c["M"])
    projs.append(_proj(main, main, own))
    tables.append(_conn(rng, c["H"], own, c["H"], c["M"]))
    more = {}
    if c["variant"] == "multi":
        pops = [dict(p, taua=F32(0.05), adgain=1.0) for p in pops]
        more = dict(variant=1, spike_buffer=25)
    net = capi.Net(pops, projs, DT, seed=seed & 0x7FFFFFFF, poisson_hz=c["hz"], max_ticks=128, **more)
    for q, ii in enumerate(tables):
        net.set_conn(q, ii, np.ones_like(ii))
    lgidx, masks = _rows(rng, c["patterns"], shapes)
    net.upload_stimuli_idx(lgidx, EPS, masks)
    s = types.SimpleNamespace(c=c, net=net, lgidx=lgidx, masks=masks, shapes=shapes, projs=len(projs))
    words = [(H * M + 31) // 32 for H, M in shapes]
    P = c["patterns"]
    s.plan, t, old = [], 1, 0.0
    for k in range(2 * P):
        n, prn = (c["train"], 1.0) if k < P else (c["recall"], 0.0)
        if n:
            s.plan.append((t, n, prn, old, k, 0 if k < P else 1))
            t, old = t + n, prn
    s.logs = [[_pinned((n, w), torch.int32).view(np.uint32) for w in words] for _, n, *_ in s.plan]
    s.checks = [[(_pinned(H, torch.int32), _pinned(H, torch.int32)) for H, _ in shapes] for p in s.plan if p[2] == 0.0]
    return s


def _run_net(s):
    net, c = s.net, s.c
    net.reset()
    if c["ticks"]:
        return _run_online(s)
    check = 0
    for (first, n, prn, old, row, mask), logs in zip(s.plan, s.logs):
        net.use_stimulus(row, mask)
        net.run(first, n, prn, old)
        for p, log in enumerate(logs):
            net.spike_log_async(p, log)
        if prn == 0.0:
            for p, (idx, cnt) in enumerate(s.checks[check]):
                net.check_count(p, 0, n)
                net.check_result_async(p, idx, cnt)
            check += 1
    net.sync()
    last = len(s.shapes) - 1
    checks = [np.concatenate([pops[p][k] for pops in s.checks for p in range(last + 1)]) for k in (0, 1)] if s.checks else []
    return dict(logs=[np.concatenate([logs[p] for logs in s.logs]) for p in range(last + 1)], checks=checks,
                wij=net.read(f"wij_{s.projs - 1}"), bj=net.read(f"bj_{last}"), counters=np.array(net.counters()))


def _run_online(s):
    net = s.net
    seen = []
    for k in range(s.c["ticks"]):
        row = s.lgidx[(k // 8) % s.c["patterns"]]
        net.set_stimulus_idx(row, EPS, s.masks[0])
        net.run(1 + k, 1, 1.0, 0.0 if k == 0 else 1.0)
        seen.append([net.spike_log(p)[0] for p in range(len(s.shapes))])
    last = len(s.shapes) - 1
    return dict(spikes=[np.stack(x) for x in zip(*seen)], dsup=net.read(f"dsup_{last}"), bj=net.read(f"bj_{last}"),
                wij=net.read(f"wij_{s.projs - 1}"))


def _work_net(c):
    mcus = (c["H0"] + c["H"]) * c["M"]
    ticks = c["ticks"] or c["patterns"] * (c["train"] + c["recall"])
    slots0 = min(c["slots"], c["H0"] * c["M"])
    slots = min(c["slots1"] if c["H0"] else c["slots"], c["H"] * c["M"])
    rate = SPIKE_RATE * (c["H0"] + c["H"]) + c["hz"] * DT * mcus  # spikes a tick, over all populations
    share = rate / mcus                                        # ... and per MCU
    rows = share * c["H"] * (slots0 + slots) * c["M"]          # row cells a tick
    cols = rows if c["variant"] == "lazy" else 0.0             # column cells a tick
    cells = c["H"] * (slots0 + slots) * c["M"]
    byt = ticks * (44 * rows + 40 * cols + 33 * mcus) + 4 * cells
    return dict(bytes=byt, flops=ticks * (40 * (rows + cols) + 60 * mcus))


# ------------------------------------------------------------------------------------------------ batches

def _members(c, seed):
    """networks with HCU and MCU counts drawn uniformly, every HCU fed by every MCU, delay 1"""
    sizes = np.random.default_rng(c["members"] * 1000003 + c["hcu_hi"] * 1009 + c["mcu_hi"])  # the work is the case's own
    hs = sizes.integers(c["hcu_lo"], c["hcu_hi"] + 1, c["members"])
    ms = sizes.integers(c["mcu_lo"], c["mcu_hi"] + 1, c["members"])
    rng = np.random.default_rng(seed)
    out = []
    for i, (H, M) in enumerate(zip(hs.tolist(), ms.tolist())):
        lgidx, masks = _rows(rng, c["patterns"], [(H, M)])
        ii = np.tile(np.arange(H * M, dtype=np.int32), H)
        out.append(types.SimpleNamespace(index=i, H=H, M=M, C=H * M, seed=(seed * 100003 + i + 1) & 0x7FFFFFFF,
                                         pop=_pop(H, M), proj=_proj(0, 0, H * M), ii=ii, di=np.ones_like(ii),
                                         lgidx=lgidx, wmask=masks))
    return out


def _prepare_batch(c, seed):
    ms = _members(c, seed)
    eng = batch.BatchEngine(ms, dt=DT, eps=EPS, max_ticks=128)
    return types.SimpleNamespace(c=c, eng=eng, n=len(ms), runs=batch.schedule(c["patterns"], c["train"], c["recall"]))


def _run_batch(s):
    s.eng.reset()
    for run in s.runs:
        s.eng.run_segment(*run)
    s.eng.sync()
    logs = [s.eng.spike_log(m).reshape(-1) for m in range(s.n)]  # of the last recall
    return dict(logs=np.concatenate(logs), bj=np.concatenate([s.eng.read(m, "bj_0") for m in range(s.n)]),
                dsup=np.concatenate([s.eng.read(m, "dsup_0") for m in range(s.n)]), counters=np.array(s.eng.counters()))


def _work_batch(c):
    ticks = c["patterns"] * (c["train"] + c["recall"])
    mcus = cells = all_cells = 0
    for m in _members(c, 0):
        mcus += m.C
        cells += SPIKE_RATE * m.H * m.C
        all_cells += m.H * m.C * m.M
    return dict(bytes=ticks * (84 * cells + 33 * mcus) + 48 * all_cells, flops=ticks * (80 * cells + 60 * mcus))


# ------------------------------------------------------------------------------------------------ replicate recall

def _recall_inputs(c, seed):
    """weights and biases like those that training leaves: co-active MCUs of some patterns excite each other, the
    others are near or below zero; the last spikes before recall; cues of a quarter of the HCUs"""
    H, M, R = c["H"], c["M"], c["R"]
    N = H * M
    rng = np.random.default_rng(seed)
    g = torch.Generator().manual_seed(seed & 0x7FFFFFFF)
    pats = rng.integers(0, M, (16, H)).astype(np.int32)
    on = torch.zeros(16, N)
    on[torch.arange(16)[:, None], torch.from_numpy(pats.astype(np.int64)) + torch.arange(H) * M] = 1
    w = torch.randn(N, N, generator=g).mul_(0.3).sub_(0.5 / H)
    w += (on.t() @ on).mul_(min(1.0, 16.0 / H))
    bj = torch.randn(N, generator=g).mul_(0.2).sub_(math.log(M))
    hist = [(rng.random(N) < SPIKE_RATE / M + 0.02).astype(np.int8) for _ in range(3)]
    cued = (H + 3) // 4
    lg = np.where(np.arange(H) < cued, pats[np.arange(R) % 16], NO_INPUT).astype(np.int32)
    wm = np.tile((np.arange(H) >= cued).astype(np.float32), (R, 1))
    return dict(w=w.numpy(), bj=bj.numpy(), epsc=np.zeros(N, np.float32),
                dsup=np.full(N, -math.log(M), np.float32), hist=hist, lg=lg, wm=wm, seed=seed & 0x7FFFFFFF)


def _prepare_recall(c, seed):
    x = _recall_inputs(c, seed)
    eng = recall.Recall(c["H"], c["M"], c["R"], _pop(c["H"], c["M"]), DT, KEPSC, seed_base=x["seed"], poisson_hz=c["hz"],
                        contraction=c["form"])
    eng.load_state(x["w"], x["bj"], x["epsc"], x["dsup"], *x["hist"])
    return types.SimpleNamespace(c=c, eng=eng, lg=x["lg"], wm=x["wm"])


def _run_recall(s):
    """one trial: cues, the ticks with the counting window over all of them, the counters (the network goes on from
    where the last trial left it)"""
    c, eng = s.c, s.eng
    eng.clear_counts()
    eng.set_cues(s.lg, EPS, s.wm)
    eng.run(1, c["ticks"], 1, c["ticks"])
    out = dict(counts=eng.read("counts"))
    if c["R"] * c["H"] * c["M"] <= 1 << 17:
        out.update(dsup=eng.read("dsup"), epsc=eng.read("epsc"), spike=eng.read("spike"))
    return out


def _work_recall(c):
    N = c["H"] * c["M"]
    rate = SPIKE_RATE / c["M"] + c["hz"] * DT
    state = c["R"] * N
    w = N * N * (2 if c["form"] == "bf16" else 4)
    # dsup and epsc are read and written each tick; W is read once; one addition per spike and destination
    return dict(bytes=c["ticks"] * 16 * state + w + state, flops=c["ticks"] * state * (rate * N + 60))


def _philox(c0, tick, k0, k1):
    """Philox4x32-10 lanes for counter (c0, tick, 0, 0); uint32 arrays in uint64"""
    M32 = np.uint64(0xFFFFFFFF)
    c = [c0.astype(np.uint64), np.full_like(c0, tick, np.uint64), np.zeros_like(c0, np.uint64), np.zeros_like(c0, np.uint64)]
    k0, k1 = k0.astype(np.uint64), np.uint64(k1)
    for r in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ k0, b & M32, (a >> np.uint64(32)) ^ c[3] ^ k1, a & M32]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & M32, (k1 + np.uint64(0xBB67AE85)) & M32
    return np.stack(c, axis=-1)


def _exact_recall(c, seed):
    """the trial in 64 bits, from the model's definition (weights rounded once where the form says so)"""
    if c["R"] * c["H"] * c["M"] > 1 << 17:
        return None
    x = _recall_inputs(c, seed)
    H, M, R, N = c["H"], c["M"], c["R"], c["H"] * c["M"]
    w = torch.from_numpy(x["w"])
    w = (w.bfloat16().double() if c["form"] == "bf16" else w.double()).numpy()
    rep = lambda v: np.tile(np.asarray(v, np.float64), (R, 1))  # noqa: E731
    dsup, epsc, bj = rep(x["dsup"]), rep(x["epsc"]), x["bj"].astype(np.float64)
    spikes = [rep(h) for h in x["hist"]]
    wm = np.repeat(x["wm"].astype(np.float64), M, axis=1)
    hit = np.repeat(x["lg"], M, axis=1) == np.tile(np.arange(M), H)
    lginp = np.where(hit, math.log(float(F32(1) + F32(EPS))), math.log(float(F32(EPS))))
    taumdt, keep = float(F32(DT) / F32(0.005)), float(F32(1) - F32(KEPSC))
    maxfqdt, pr = float(F32(100.0) * F32(DT)), float(F32(c["hz"]) * F32(DT))
    quad = np.tile(np.arange(N // 4), (R, 1))
    keys = (x["seed"] + np.arange(R))[:, None]
    u01 = lambda t, stream: (_philox(quad, t, keys, stream).reshape(R, N) >> np.uint64(8)) * 2.0 ** -24  # noqa: E731
    for t in range(1, c["ticks"] + 1):
        sup = float(F32(LGBIAS)) + lginp + wm * (bj + epsc)
        dsup = dsup + (sup - dsup) * taumdt
        d = dsup.reshape(R, H, M)
        mx = np.maximum(dsup[:, :1], d.max(axis=2))[:, :, None]
        act = np.exp(d - mx) * np.minimum(1.0, np.exp(mx))
        total = act.sum(axis=2, keepdims=True)
        act = (act / np.maximum(1.0, total)).reshape(R, N)
        s = u01(t, 0) < act * maxfqdt
        if c["hz"] > 0:
            s |= u01(t, 2) < pr
        epsc = epsc * keep + spikes[-3] @ w
        spikes.append(s.astype(np.float64))
    return dict(counts=None, dsup=dsup, epsc=epsc, spike=None)


# ------------------------------------------------------------------------------------------------ by kind

def prepare(case, seed):
    return dict(net=_prepare_net, batch=_prepare_batch, recall=_prepare_recall)[case["kind"]](case, seed)


def run(state):
    return dict(net=_run_net, batch=_run_batch, recall=_run_recall)[state.c["kind"]](state)


def work(case):
    return dict(net=_work_net, batch=_work_batch, recall=_work_recall)[case["kind"]](case)


def exact(case, seed):
    """None for networks with plasticity: their state is defined by the reference's own sequence of FP32 operations (its
    closed-form decays cancel between near-equal time constants, far from what 64 bits give), and later spikes depend on it"""
    return _exact_recall(case, seed) if case["kind"] == "recall" else None
