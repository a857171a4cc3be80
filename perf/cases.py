"""Workloads of the framework through its public entry points, for timing it.

Every case is a dict of plain values; `prepare` makes from it (and a seed) what a user's program
has in hand before the call - streams, a loaded bank, a filled cache, a scheduler, a network -
and `run` is one pass of the user's work, with the outputs the user reads back.

Outputs are those that one input determines. Transfers move fixed amounts between accounts whose
funds never run short, so the final balances do not depend on the commit order; the sums of
read-only rounds that run between transfers do, and are read back only where the reads follow
the transfers (audits) or run in stream order (the lanes). Cached values are functions of their
keys, as refreshes of unchanged content are, and every key that is SET is in the table.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "csmv-gpu-stm_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import csmv_gb300 as cg  # noqa: E402

FUNDS = 100_000_000   # opening balance of the order-independent banks
OPENING = 1000        # opening balance where the order is fixed: funds do run short there


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------

def _bank(**kw):
    c = dict(kind="bank", accounts=1 << 20, rounds=1 << 15, dist="uniform", ro_pct=20, ro_reads=32,
             up_reads=4, amt=1, method=3, depth=8, warps=12, ctas=0, max_reads=0, host=False,
             audit=False)
    c.update(kw)
    return c


def listed():
    return [
        # an interactive call: one small stream from host buffers on a default handle, then the
        # balances; launches, copies and the hand-offs of a handful of rounds are all of it
        _bank(name="bank_small_call", accounts=4096, rounds=32, ro_pct=10, ro_reads=8, up_reads=2,
              amt=10, method=1, depth=4, warps=15, host=True),
        # the plain small bank: 4096 accounts, 8 blocks x 128 client threads x 256 transactions,
        # 90 % transfers of 1..10, 10 % sums of 8, host buffers, per-transaction commit
        _bank(name="bank_plain", accounts=4096, rounds=8192, ro_pct=10, ro_reads=8, up_reads=2,
              amt=10, method=1, depth=4, warps=4, ctas=8, host=True),
        # the bank at scale without contention: 2^20 accounts, a 2^20-transaction batch resident
        # on the device, transfers reading 4 and writing 2, 20 % scans of 32, group commit
        _bank(name="bank_uniform", max_reads=4),
        # ragged sizes and a hot region (1 % of the accounts draw 30 %), per-transaction commit,
        # then an audit: read-only rounds over every account, whose sums are read back
        _bank(name="bank_hotspot_audit", accounts=300007, rounds=9999, dist="hotspot",
              ro_reads=13, up_reads=5, method=1, depth=4, warps=15, audit=True),
        # the contended bank, Zipf(0.99), group commit in stream order (no scheduler)
        _bank(name="bank_zipf", rounds=4096, dist="zipf", max_reads=4),
        # the contended bank behind the learned scheduler: probe, train, plan, run
        dict(name="sched_zipf", kind="sched", accounts=1 << 20, rounds=1 << 15, dist="zipf",
             ro_pct=20, ro_reads=32, up_reads=4),
        # transactions known to conflict, run in stream order by the serial lane
        dict(name="serial_lane", kind="lane", lane="serial", accounts=1 << 20, rounds=1024,
             dist="zipf", ro_pct=20, ro_reads=32, up_reads=4, depth=8),
        # ... and by the dataflow lane
        dict(name="flow_lane", kind="lane", lane="flow", accounts=1 << 20, rounds=8192,
             dist="zipf", ro_pct=20, ro_reads=32, up_reads=4, depth=8),
        # one batch of the transactional cache from host buffers: 64 K requests, 99 % GET,
        # Zipf(0.99) keys over 4 M, the most popular 2^20 of them stored
        dict(name="cache_batch", kind="cache", sets=1 << 20, keys=1 << 22, stored=1 << 20,
             rounds=2048, get_pct=99),
        # a serving session: batches of 1 K to 64 K requests submitted as room allows, 95 % GET
        dict(name="cache_serve", kind="serve", sets=1 << 20, keys=1 << 22, stored=1 << 20,
             batches=12, get_pct=95),
        # the conflict predictor over a whole batch of 2^20 transactions
        dict(name="predict", kind="predict", n=1 << 20),
        # one training step on the default probe slice (5 % of 2^20): gradient and Adam
        dict(name="train_step", kind="train", n=52448),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["bank"] * 4 + ["sched", "sched", "lane", "lane", "cache", "serve",
                                      "predict", "train"])
    if kind == "bank":
        dist = rng.choice(["uniform", "uniform", "hotspot", "zipf"])
        method = 3 if dist == "zipf" else rng.choice([1, 3])
        up = rng.choice([2, 3, 4, 5, 8])
        return _bank(accounts=size(4096 if dist == "uniform" else 1 << 16, 1 << 20),
                     rounds=size(8, 4096 if dist == "zipf" else 1 << 15), dist=dist,
                     ro_pct=rng.choice([0, 10, 20, 50]), ro_reads=rng.randint(1, 32), up_reads=up,
                     amt=rng.randint(1, 10) if up == 2 else 1, method=method,
                     depth=rng.choice([4, 8]), warps=rng.choice([4, 8, 12, 15]),
                     max_reads=4 if up <= 4 and rng.random() < 0.5 else 0,
                     host=rng.random() < 0.4, audit=rng.random() < 0.25)
    if kind == "sched":
        return dict(kind="sched", accounts=size(1 << 17, 1 << 20), rounds=size(512, 1 << 15),
                    dist=rng.choice(["zipf", "hotspot"]), ro_pct=rng.choice([0, 10, 20, 50]),
                    ro_reads=rng.randint(1, 32), up_reads=rng.randint(2, 4))
    if kind == "lane":
        lane = rng.choice(["serial", "flow"])
        return dict(kind="lane", lane=lane, accounts=size(1 << 12, 1 << 20),
                    rounds=size(8, 1024 if lane == "serial" else 8192),
                    dist=rng.choice(["uniform", "zipf", "hotspot"]),
                    ro_pct=rng.choice([0, 10, 20]), ro_reads=rng.randint(1, 32),
                    up_reads=rng.randint(2, 8), depth=rng.choice([4, 8]))
    if kind in ("cache", "serve"):
        sets = size(1 << 17, 1 << 20)
        c = dict(kind=kind, sets=sets, keys=4 * sets, stored=sets, get_pct=rng.choice([90, 95, 99]))
        c.update(dict(rounds=size(1, 2048)) if kind == "cache" else dict(batches=rng.randint(2, 12)))
        return c
    return dict(kind=kind, n=size(1000, 1 << 20 if kind == "predict" else 60000))


# ---------------------------------------------------------------------------------------------
# streams
# ---------------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _zipf_cdf(n, theta=0.99):
    w = torch.arange(1, n + 1, device="cuda", dtype=torch.float64).pow_(-theta).cumsum_(0)
    return w / w[-1].clone()


def _accounts(c, shape, g):
    """Account choices [shape] of the case's distribution: int64, on the device."""
    n = c["accounts"]
    if c["dist"] == "zipf":
        u = torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)
        return torch.searchsorted(_zipf_cdf(n), u).clamp_(max=n - 1)
    a = torch.randint(0, n, shape, generator=g, device="cuda")
    if c["dist"] == "hotspot":  # 1 % of the accounts, a region somewhere, draw 30 %
        hot_n = max(1, n // 100)
        base = int(torch.randint(0, n, (1,), generator=g, device="cuda"))
        h = (torch.randint(0, hot_n, shape, generator=g, device="cuda") + base) % n
        a = torch.where(torch.rand(shape, generator=g, device="cuda") < 0.3, h, a)
    return a


def _stream(c, seed, kind, amt):
    """(op, off, addr) int32 device tensors: rounds of 32 transactions, each round transfers of
    distinct accounts or read-only sums, in the library's stream format."""
    g = _gen(seed)
    R, ro_reads, up = c["rounds"], c["ro_reads"], c["up_reads"]
    ro = torch.rand(R, generator=g, device="cuda") < c["ro_pct"] / 100
    ro = ro.repeat_interleave(32)
    n = R * 32
    amt0 = torch.randint(1, amt + 1, (n,), generator=g, device="cuda")
    op = torch.where(ro, 0 | (ro_reads << 2) | (1 << 8) | (1 << 20),
                     kind | (up << 2) | (amt0 << 8) | (amt << 20))
    reads = torch.where(ro, ro_reads, up)
    off = reads.cumsum(0) - reads
    addr = torch.empty(int(reads.sum()), dtype=torch.int64, device="cuda")
    t_up = (~ro).nonzero().squeeze(1)
    a = _accounts(c, (t_up.numel(), up), g)
    for _ in range(12):  # a transfer's accounts are distinct: draw repeated ones again
        dup = torch.zeros_like(a, dtype=torch.bool)
        for k in range(1, up):
            dup[:, k] = (a[:, :k] == a[:, k:k + 1]).any(1)
        rows = dup.any(1).nonzero().squeeze(1)
        if rows.numel() == 0:
            break
        a[rows] = torch.where(dup[rows], _accounts(c, (rows.numel(), up), g), a[rows])
    addr[off[t_up][:, None] + torch.arange(up, device="cuda")] = a
    t_ro = ro.nonzero().squeeze(1)
    if t_ro.numel():
        addr[off[t_ro][:, None] + torch.arange(ro_reads, device="cuda")] = \
            _accounts(c, (t_ro.numel(), ro_reads), g)
    return [t.to(torch.int32) for t in (op, off, addr)]


def _audit(accounts):
    """Read-only rounds that sum every account once, up to 32 accounts per transaction."""
    n = -(-accounts // (32 * 32)) * 32
    t = torch.arange(n, device="cuda")
    lo = t * 32
    reads = (accounts - lo).clamp(1, 32)  # padding transactions read the last account
    off = torch.minimum(lo, torch.full_like(lo, accounts - 1))
    op = (reads << 2) | (1 << 8) | (1 << 20)
    return [x.to(torch.int32) for x in (op, off, torch.arange(accounts, device="cuda"))]


def _dev_stream(t):
    return cg.BankStream(t[0].numel(), t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(),
                         t[2].numel())


def _host_stream(t):
    return cg.Stream(*[x.cpu().numpy().view(np.uint32) for x in t])


# ---------------------------------------------------------------------------------------------
# cache requests
# ---------------------------------------------------------------------------------------------

def _mix(x):
    x = (x ^ (x >> np.uint32(16))) * np.uint32(0x85EBCA6B)
    x = (x ^ (x >> np.uint32(13))) * np.uint32(0xC2B2AE35)
    return x ^ (x >> np.uint32(16))


def _requests(ids, is_set, seed):
    """Requests for key ids: 16-byte keys, 32-byte values that are functions of the key."""
    ids = ids.astype(np.uint32)
    with np.errstate(over="ignore"):
        key = np.stack([ids] + [_mix(ids * np.uint32(4) + np.uint32(j)) for j in (1, 2, 3)], axis=1)
        val = np.stack([_mix(ids * np.uint32(8) + np.uint32(j) + np.uint32(seed * 2654435761 & 0xFFFFFFFF))
                        for j in range(8)], axis=1)
    val[~is_set] = 0
    return cg.Requests(np.where(is_set, cg.MEMCD_SET, cg.MEMCD_GET).astype(np.uint32),
                       np.ascontiguousarray(key), np.ascontiguousarray(val))


def _stored_ids(c):
    """The most popular ids that fill no set: every one of them stays stored."""
    ids = np.arange(c["stored"], dtype=np.uint32)
    key = _requests(ids, np.zeros(len(ids), bool), 0).key
    with np.errstate(over="ignore"):
        h = (key[:, 0] * np.uint32(0x9E3779B1) ^ key[:, 1] * np.uint32(0x85EBCA6B) ^
             key[:, 2] * np.uint32(0xC2B2AE35) ^ key[:, 3] * np.uint32(0x27D4EB2F))
        h ^= h >> np.uint32(16)
    s = h % np.uint32(c["sets"])
    load = np.bincount(s, minlength=c["sets"])
    ids = ids[load[s] <= cg.MEMCD_WAYS]
    return ids[:len(ids) // 32 * 32]


def _traffic(c, rounds, stored, g, seed):
    """A request batch: rounds of GETs over all keys or of SETs of stored keys, Zipf(0.99)."""
    n = rounds * 32
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    ids = torch.searchsorted(_zipf_cdf(c["keys"]), u).clamp_(max=c["keys"] - 1).cpu().numpy()
    is_set = (torch.rand(rounds, generator=g, device="cuda") >= c["get_pct"] / 100)
    is_set = is_set.repeat_interleave(32).cpu().numpy()
    ok = np.zeros(c["keys"], bool)
    ok[stored] = True
    back = stored[ids % len(stored)]
    return _requests(np.where(is_set & ~ok[ids], back, ids), is_set, seed)


def _fills(stored, seed, step=1 << 15):
    return [_requests(stored[i:i + step], np.ones(len(stored[i:i + step]), bool), seed)
            for i in range(0, len(stored), step)]


def _batch_rounds(c):
    """Uneven batch sizes, 1 K to 64 K requests in rounds of 32."""
    return np.random.RandomState(c["batches"]).randint(32, 2049, c["batches"]).tolist()


def _collect(srv, bid):
    while True:
        r = srv.poll(bid)
        if r is not None:
            return r[0], r[1]


def _serve(srv, batches):
    """Submits the batches in order, collecting the oldest whenever admission refuses one."""
    ids, out = [], []
    for b in batches:
        while True:
            bid = srv.submit(b)
            if bid is not None:
                break
            out.append(_collect(srv, ids[len(out)]))
        ids.append(bid)
    while len(out) < len(ids):
        out.append(_collect(srv, ids[len(out)]))
    return out


# ---------------------------------------------------------------------------------------------
# network inputs
# ---------------------------------------------------------------------------------------------

def _features(n, seed):
    """Thermometer-coded indicators like the scheduler's (three 16-level counts, two 8-level
    rates), bf16 [n, 64], and labels that depend on them."""
    g = _gen(seed)
    cols = []
    level = []
    for width in (16, 16, 16, 8, 8):
        lv = (torch.rand(n, generator=g, device="cuda").pow(2) * (width + 1)).long()
        level.append(lv.float() / width)
        cols.append(lv[:, None] > torch.arange(width, device="cuda"))
    x = torch.cat(cols, 1).to(torch.bfloat16)
    risk = 0.45 * level[0] + 0.45 * level[1] + 0.2 * level[3]
    y = (risk + 0.3 * torch.rand(n, generator=g, device="cuda") > 0.6).float()
    return x.contiguous(), y


def _params(seed):
    """Network weights with nonzero biases (fp32 parameter block)."""
    r = np.random.RandomState(seed % (1 << 31))
    p = np.zeros(cg.MLP_PARAMS, np.float32)
    o = 0
    for n, b in ((64 * 128, 1 / 8), (128, 0.1), (128 * 128, 1 / 128 ** 0.5), (128, 0.1),
                 (128, 1 / 128 ** 0.5), (1, 0.1)):
        p[o:o + n] = r.uniform(-b, b, n)
        o += n
    return p


# ---------------------------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------------------------

def prepare(case, seed):
    c = case
    s = {"case": c}
    if c["kind"] == "bank":
        t = _stream(c, seed, cg.KIND_TRANSFER, c["amt"])
        audit = _audit(c["accounts"]) if c["audit"] else None
        n = max(t[0].numel(), audit[0].numel() if audit else 0)
        s["bank"] = cg.Bank(n_accounts=c["accounts"], init_value=FUNDS, version_depth=c["depth"],
                            client_warps=c["warps"], ctas=c["ctas"], prevalidate=c["method"],
                            max_reads=c["max_reads"], max_txn=n)
        s["bank"].load()
        if c["host"]:
            s["stream"], s["audit"] = _host_stream(t), _host_stream(audit) if audit else None
        else:
            s["keep"] = (t, audit)
            s["stream"], s["audit"] = _dev_stream(t), _dev_stream(audit) if audit else None
    elif c["kind"] == "sched":
        t = _stream(c, seed, cg.KIND_TRANSFER, 1)
        n = t[0].numel()
        s["bank"] = cg.Bank(n_accounts=c["accounts"], init_value=FUNDS, version_depth=8,
                            client_warps=12, prevalidate=3, max_reads=4, max_txn=n)
        s["bank"].load()
        s["sched"] = cg.Scheduler(n_accounts=c["accounts"], max_txn=n, plan=1, probe_rounds_pct=2,
                                  probe_every=3)
        s["keep"], s["stream"] = t, _dev_stream(t)
    elif c["kind"] == "lane":
        t = _stream(c, seed, cg.KIND_TRANSFER, 10)
        s["bank"] = cg.Bank(n_accounts=c["accounts"], init_value=OPENING, version_depth=c["depth"],
                            max_txn=t[0].numel())
        s["bank"].load()
        s["keep"], s["stream"], s["ts"] = t, _dev_stream(t), 0
    elif c["kind"] == "cache":
        stored, g = _stored_ids(c), _gen(seed)
        s["cache"] = cg.Memcd(n_sets=c["sets"], max_req=max(1 << 15, c["rounds"] * 32))
        for f in _fills(stored, seed):
            s["cache"].run(f)
        s["req"] = _traffic(c, c["rounds"], stored, g, seed)
    elif c["kind"] == "serve":
        stored, g = _stored_ids(c), _gen(seed)
        s["srv"] = cg.Server(n_sets=c["sets"], arena_requests=1 << 18, max_inflight_sets=1 << 16)
        s["srv"].start()
        _serve(s["srv"], _fills(stored, seed))
        s["srv"].stop()
        s["req"] = [_traffic(c, r, stored, g, seed) for r in _batch_rounds(c)]
    else:
        s["x"], s["y"] = _features(c["n"], seed)
        s["net"] = cg.Mlp(seed=1)
        s["net"].set_params(_params(seed))
        s["p"] = torch.empty(c["n"], dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    return s


def run(state):
    c = state["case"]
    if c["kind"] == "bank":
        bank = state["bank"]
        go = bank.run if c["host"] else bank.run_device
        st = go(state["stream"])
        out = {"commits": [st.commits_update, st.commits_readonly, st.commits_nowrite]}
        if c["audit"]:
            go(state["audit"])
            n = -(-c["accounts"] // 1024) * 32
            out["audit"] = bank.results(n)[1]
        out["values"] = bank.values()
        return out
    if c["kind"] == "sched":
        rep = state["sched"].run(state["bank"], state["stream"])
        return {"commits": rep.commits, "values": state["bank"].values()}
    if c["kind"] == "lane":
        bank = state["bank"]
        st = (bank.run_serial_device if c["lane"] == "serial" else bank.run_flow_device)(
            state["stream"])
        used, state["ts"] = st.final_ts - state["ts"], st.final_ts
        n = c["rounds"] * 32
        log = np.full(n, cg.HOLE, np.uint32)
        log[:used], outcome, result = bank.log(n, used)
        return {"log": log, "outcome": outcome, "result": result, "values": bank.values()}
    if c["kind"] == "cache":
        found, val, st = state["cache"].run(state["req"])
        return {"found": found, "value": val, "commits": st.commits}
    if c["kind"] == "serve":
        srv = state["srv"]
        srv.start()
        got = _serve(srv, state["req"])
        st = srv.stop()
        return {"found": [f for f, _ in got], "value": [v for _, v in got], "commits": st.commits}
    if c["kind"] == "predict":
        state["net"].forward(c["n"], state["x"].data_ptr(), state["p"].data_ptr())
        return state["p"]
    net = state["net"]
    loss = net.grad(c["n"], state["x"].data_ptr(), state["y"].data_ptr())
    grads = net.grads()
    net.adam_step(3e-3)
    return {"loss": np.float32(loss), "grads": grads, "params": net.params()}


# ---------------------------------------------------------------------------------------------
# work and exact results
# ---------------------------------------------------------------------------------------------

def work(case):
    c = case
    if c["kind"] in ("bank", "sched", "lane"):
        # the stream once (8 B a transaction, 4 B an access), 8 B for each version read or
        # written, the balances (and, for the lanes, log, outcomes and results) out
        n = c["rounds"] * 32
        ro = n * c["ro_pct"] / 100
        reads = ro * c["ro_reads"] + (n - ro) * c["up_reads"]
        b = n * 8 + reads * 12 + (n - ro) * 16 + c["accounts"] * 4
        if c["kind"] == "lane":
            b += n * 12
        if c.get("audit"):
            b += c["accounts"] * 12.75
        return {"bytes": b, "flops": 0}
    if c["kind"] in ("cache", "serve"):
        # request in (kind, key, SET value), the set's tags and the record, result out
        n = 32 * (c["rounds"] if c["kind"] == "cache" else sum(_batch_rounds(c)))
        return {"bytes": n * (4 + 16 + 128 + 64 + 36) + n * (100 - c["get_pct"]) / 100 * 104,
                "flops": 0}
    macs = 64 * 128 + 128 * 128 + 128
    if c["kind"] == "predict":
        return {"bytes": c["n"] * 132 + cg.MLP_PARAMS * 2, "flops": 2 * macs * c["n"]}
    # forward, weight gradients, and the gradient through the second layer
    return {"bytes": c["n"] * 132 + cg.MLP_PARAMS * 4 * 8,
            "flops": (4 * macs + 2 * (128 * 128 + 128)) * c["n"]}


def _exact_net(p, x):
    o = np.cumsum([0, 64 * 128, 128, 128 * 128, 128, 128, 1])
    w = [torch.from_numpy(p[a:b]).cuda() for a, b in zip(o[:-1], o[1:])]
    w = [t.to(torch.bfloat16).double() if i % 2 == 0 else t.double() for i, t in enumerate(w)]
    h1 = (x @ w[0].view(64, 128) + w[1]).relu()
    h2 = (h1 @ w[2].view(128, 128) + w[3]).relu()
    return w, h1, h2, h2 @ w[4] + w[5]


def exact(case, seed):
    """The network in 64 bits on the bf16 weights; every other output is whole numbers."""
    c = case
    if c["kind"] not in ("predict", "train"):
        return None
    x, y = _features(c["n"], seed)
    p0 = _params(seed)
    x, y = x.double(), y.double()
    w, h1, h2, z = _exact_net(p0, x)
    if c["kind"] == "predict":
        return torch.sigmoid(z)
    n = c["n"]
    loss = (z.clamp(min=0) - y * z + torch.log1p(torch.exp(-z.abs()))).mean()
    dz = (torch.sigmoid(z) - y) / n
    d2 = dz[:, None] * w[4] * (h2 > 0)
    d1 = (d2 @ w[2].view(128, 128).t()) * (h1 > 0)
    g = torch.cat([(x.t() @ d1).reshape(-1), d1.sum(0), (h1.t() @ d2).reshape(-1), d2.sum(0),
                   h2.t() @ dz, dz.sum()[None], torch.zeros(3, dtype=torch.float64, device="cuda")])
    g = g.cpu().numpy()
    step = 3e-3 * g / (np.abs(g) + 1e-8)  # the first Adam step: mean and root cancel but for eps
    return {"loss": np.float64(loss.item()), "grads": g, "params": p0.astype(np.float64) - step}
