"""Performance cases: the work a user has this generator do, through the public Python entry points.

Every case is one call pattern of real use: single values, device arrays of each output kind from
a few values to 2^30, host arrays, jumps of many offsets, batches of independent streams and a
server's draw requests.  ``listed`` names the fixed ones, ``draw`` gives more of the same ranges,
``prepare`` makes what a program has in hand before the call (handles, plans, buffers), ``run`` is
one pass, ``work`` the bytes it cannot do without and ``exact`` the same outputs from plain torch.
"""
import math

import numpy as np
import torch

import mrg8_gb300 as m
from mrg8_gb300 import api, serve

P = 2147483647
COEF = (1089656042, 1906537547, 1764115693, 1304127872, 189748160, 1984088114, 626062218, 1927846343)
KINDS = {"u32": m.U32, "f64_original": m.F64_ORIGINAL, "f64_shifted": m.F64_SHIFTED,
         "f32_original": m.F32_ORIGINAL, "f32_shifted": m.F32_SHIFTED}
DTYPES = {"u32": torch.int32, "f64_original": torch.float64, "f64_shifted": torch.float64,
          "f32_original": torch.float32, "f32_shifted": torch.float32}
BYTES = {"u32": 4, "f64_original": 8, "f64_shifted": 8, "f32_original": 4, "f32_shifted": 4}
MIX = ("f64_shifted", "f32_shifted", "u32")


def listed():
    return [
        # A program that takes its uniforms one at a time on the host, as rand() of the reference's host class.
        {"name": "one value", "op": "value"},
        # A kernel's worth of random numbers for a small simulation step.
        {"name": "device f64 1000", "op": "device", "kind": "f64_original", "n": 1000, "skip": 0},
        # Integers into the middle of a larger array (its start on no 16-byte boundary), an odd count.
        {"name": "device u32 100003 ragged", "op": "device", "kind": "u32", "n": 100003, "skip": 1},
        # One layer's worth of fp32 noise.
        {"name": "device f32 5000001", "op": "device", "kind": "f32_shifted", "n": 5000001, "skip": 0},
        # The 2^24 uniforms of the single-stream comparison with the sequential class.
        {"name": "device f64 2^24", "op": "device", "kind": "f64_original", "n": 1 << 24, "skip": 0},
        # The bulk workload: 2^30 uniforms from one seed, fp64 in the CUDA class's scaling and fp32.
        {"name": "device f64 2^30", "op": "device", "kind": "f64_shifted", "n": 1 << 30, "skip": 0},
        {"name": "device f32 2^30", "op": "device", "kind": "f32_shifted", "n": 1 << 30, "skip": 0},
        # Uniforms for a host program (pinned memory), as the reference's host calls return them.
        {"name": "host f64 2^24", "op": "host", "kind": "f64_original", "n": 1 << 24},
        # Start states of 65,536 substreams at arbitrary places of the stream.
        {"name": "jumps 65536", "op": "jumps", "count": 65536, "bits": 63},
        # The same 65,536 substreams with 4,096 integers each, in one batch.
        {"name": "batch 65536 x 4096 u32", "op": "batch", "count": 65536, "low": 4096, "high": 4096, "kinds": "u32",
         "bits": 63},
        # Ten thousand independent generators of uneven lengths and mixed kinds in one launch.
        {"name": "batch 10000 uneven", "op": "batch", "count": 10000, "low": 1, "high": 1 << 22, "kinds": "mix",
         "bits": 0},
        # A burst of draw requests to a server, results read back to the host.
        {"name": "serve 48 requests", "op": "serve", "count": 48, "low": 256, "high": 1 << 18},
    ]


def _spread(rng, low, high):
    """Log-uniform whole number in [low, high], odd ones among them."""
    return max(low, min(high, int(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng):
    op = rng.choice(("device", "device", "device", "host", "jumps", "batch", "batch", "serve"))
    kind = rng.choice(tuple(KINDS))
    if op == "device":
        return {"op": op, "kind": kind, "n": _spread(rng, 1, 1 << 30), "skip": rng.randrange(4)}
    if op == "host":
        return {"op": op, "kind": kind, "n": _spread(rng, 1, 1 << 24)}
    if op == "jumps":
        return {"op": op, "count": _spread(rng, 1, 65536), "bits": rng.randrange(1, 64)}
    if op == "batch":
        count = _spread(rng, 2, 65536)
        high = _spread(rng, 16, min(1 << 22, (1 << 31) // count))
        return {"op": op, "count": count, "low": rng.choice((1, high)), "high": high,
                "kinds": rng.choice(("mix",) + tuple(KINDS)), "bits": rng.choice((0, 20, 48, 63))}
    return {"op": op, "count": _spread(rng, 2, 64), "low": 256, "high": _spread(rng, 256, 1 << 18)}


def _streams(case, seed):
    """[(stream seed, outputs skipped, outputs, kind)] of a batch or serve case: lengths and kinds are the
    case's, the streams the seed's."""
    count, low, high = case["count"], case["low"], case["high"]
    rng = np.random.default_rng([count, low, high])
    n = np.exp(rng.uniform(np.log(low), np.log(high + 1), count)).astype(np.int64).clip(low, high)
    names = [MIX[i] for i in rng.integers(0, 3, count)]
    rng = np.random.default_rng(seed)
    seeds = rng.integers(1, 1 << 32, count)
    if case["op"] == "serve":
        offsets = rng.integers(0, 1 << 48, count)
    else:
        names = names if case["kinds"] == "mix" else [case["kinds"]] * count
        offsets = rng.integers(0, 1 << case["bits"], count, dtype=np.uint64) if case["bits"] else np.zeros(count, np.uint64)
    return [(int(s), int(o), int(k), d) for s, o, k, d in zip(seeds, offsets, n, names)]


def _layout(streams):
    """Each stream's place in one array of its kind (starts on 16 bytes, as an allocator gives them), and the
    arrays' sizes."""
    size, place = {}, []
    for _, _, n, kind in streams:
        at = size.get(kind, 0)
        place.append((kind, at))
        size[kind] = at + -(-n // 4) * 4
    return place, size


def prepare(case, seed):
    op = case["op"]
    if op in ("value", "device", "host"):
        g = m.MRG8(seed + 1)
        if op == "value":
            return {"case": case, "g": g}
        kind = case["kind"]
        if op == "host":
            out = torch.empty(case["n"], dtype=DTYPES[kind], pin_memory=True)
        else:
            out = torch.empty(case["n"] + case["skip"], dtype=DTYPES[kind], device="cuda")[case["skip"]:]
        return {"case": case, "g": g, "out": out, "kind": kind}
    if op == "jumps":
        rng = np.random.default_rng(seed)
        offsets = rng.integers(0, 1 << case["bits"], case["count"], dtype=np.int64)
        return {"case": case, "state": api.seed_state(seed + 1), "offsets": torch.from_numpy(offsets).cuda()}
    streams = _streams(case, seed)
    if op == "batch":
        place, size = _layout(streams)
        out = {k: torch.zeros(v, dtype=DTYPES[k], device="cuda") for k, v in size.items()}
        insts = [(api.seed_state(s), o, out[kind][at:at + n], KINDS[kind])
                 for (s, o, n, _), (kind, at) in zip(streams, place)]
        return {"case": case, "out": out, "batch": m.Batch(insts)}
    srv = serve.Server(budget_bytes=256 << 20)
    # Every fourth request draws from a generator that the server keeps.
    gens = [srv.add_generator(api.seed_state(seed + 1 + k)) for k in range(4)]
    asked = [{"n": n, "kind": KINDS[d], "generator": gens[(i // 4) % 4]} if i % 4 == 0 else
             {"n": n, "kind": KINDS[d], "seed": s, "offset": o} for i, (s, o, n, d) in enumerate(streams)]
    return {"case": case, "srv": srv, "asked": asked}


def run(state):
    op = state["case"]["op"]
    if op == "value":
        return state["g"].rand()
    if op in ("device", "host"):
        g, out, kind = state["g"], state["out"], state["kind"]
        if kind == "u32":
            return g.randint(out)
        scaling = m.ORIGINAL if kind.endswith("original") else m.SHIFTED
        return g.rand(out, scaling=scaling) if kind.startswith("f64") else g.rand_f32(out, scaling=scaling)
    if op == "jumps":
        return api.jump_states(state["state"], state["offsets"])
    if op == "batch":
        state["batch"].launch()
        return state["out"]
    srv = state["srv"]
    ticket = [srv.submit(**a) for a in state["asked"]]
    got = {}
    while len(got) < len(ticket):
        for c in srv.poll(256, 1000):
            got[c["ticket"]] = srv.read(c)
            srv.release(c["ticket"])
    return [got[t] for t in ticket]


def work(case):
    """Each output written once (and each offset read); the streams' few words of state are not counted."""
    op = case["op"]
    if op == "value":
        return {"bytes": 8, "flops": 0}
    if op in ("device", "host"):
        return {"bytes": case["n"] * BYTES[case["kind"]], "flops": 0}
    if op == "jumps":
        return {"bytes": case["count"] * 40, "flops": 0}
    return {"bytes": sum(n * BYTES[kind] for _, _, n, kind in _streams(case, 1)), "flops": 0}


# ------------------------------------------------------------------- the same outputs from plain torch


def _seeded(seed):
    x, st = (seed & 0xFFFFFFFF) or 97531, []
    for _ in range(8):
        x = 6364136223846793005 * x % (1 << 64)
        st.append(x >> 33)
    return st


def _mul(a, b):
    return [[sum(a[r][q] * b[q][c] for q in range(8)) % P for c in range(8)] for r in range(8)]


def _jumped(states, offsets):
    """Rows of `states` (int64, residues) advanced by `offsets` (whole numbers below 2^64) steps."""
    mat = [list(COEF)] + [[int(c == r) for c in range(8)] for r in range(7)]
    bits = torch.from_numpy(np.asarray(offsets, dtype=np.uint64).view(np.int64)).to(states.device)
    for i in range(64):
        on = ((bits >> i) & 1).nonzero().squeeze(1)
        if on.numel():
            a = torch.tensor(mat, dtype=torch.int64, device=states.device)
            for part in on.split(1 << 18):
                states[part] = (states[part][:, None, :] * a % P).sum(2) % P
        mat = _mul(mat, mat)
    return states


def _values(streams):
    """S of each (seed, skipped, outputs), one after another, as int64 in [1, P]."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    length = max(1, min(4096, max(n for _, _, n in streams)))
    count = np.array([-(-n // length) for _, _, n in streams])
    base = torch.tensor([_seeded(s) for s, _, _ in streams], dtype=torch.int64, device=dev)
    start = np.concatenate([np.uint64(o) + np.arange(c, dtype=np.uint64) * np.uint64(length)
                            for (_, o, _), c in zip(streams, count)])
    owner = torch.from_numpy(np.repeat(np.arange(len(streams)), count)).to(dev)
    have = np.concatenate([np.minimum(length, n - np.arange(c, dtype=np.int64) * length)
                           for (_, _, n), c in zip(streams, count)])
    st = _jumped(base[owner], start)
    a = torch.tensor(COEF, dtype=torch.int64, device=dev)
    got = []
    step = max(1, (1 << 28) // length)
    for at in range(0, len(start), step):
        lag, rows = st[at:at + step].t().contiguous(), []  # lag[0] is the newest
        k = torch.from_numpy(have[at:at + step]).to(dev)
        out = torch.empty(lag.shape[1], length, dtype=torch.int32, device=dev)
        order = list(range(8))
        for j in range(length):
            order = order[-1:] + order[:-1]
            v = (lag * a[[(i - order[0] - 1) % 8 for i in range(8)]][:, None] % P).sum(0) % P
            lag[order[0]] = v
            rows.append(torch.where(v == 0, P, v).to(torch.int32))
            if len(rows) == 64 or j == length - 1:
                out[:, j + 1 - len(rows):j + 1] = torch.stack(rows, 1)
                rows = []
        got.append(out[torch.arange(length, device=dev)[None, :] < k[:, None]])
    return torch.cat(got)


def _as_kind(s, kind):
    if kind == "u32":
        return s
    return (s.double() if kind.endswith("original") else (s - 1).double()) * (1.0 / P)


def exact(case, seed):
    op = case["op"]
    if op == "value":
        return float(_as_kind(_values([(seed + 1, 0, 1)]), "f64_original")[0])
    if op in ("device", "host"):
        return _as_kind(_values([(seed + 1, 0, case["n"])]), case["kind"])
    if op == "jumps":
        offsets = np.random.default_rng(seed).integers(0, 1 << case["bits"], case["count"], dtype=np.int64)
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        st = torch.tensor([_seeded(seed + 1)], dtype=torch.int64, device=dev).repeat(len(offsets), 1)
        st = _jumped(st, offsets.astype(np.uint64))
        return torch.where(st == 0, P, st).to(torch.int32)
    streams = _streams(case, seed)
    if op == "batch":
        place, size = _layout(streams)
        out = {}
        for kind, total in size.items():
            mine = [(s, at) for s, (k, at) in zip(streams, place) if k == kind]
            v = _as_kind(_values([s[:3] for s, _ in mine]), kind)
            full = torch.zeros(total, dtype=v.dtype, device=v.device)
            done = 0
            for (_, _, n, _), at in mine:
                full[at:at + n] = v[done:done + n]
                done += n
            out[kind] = full
        return out
    drawn, asked = [0] * 4, []
    for i, (s, o, n, kind) in enumerate(streams):
        if i % 4 == 0:
            g = (i // 4) % 4
            s, o = seed + 1 + g, drawn[g]
            drawn[g] += n
        asked.append((s, o, n))
    v, done, out = _values(asked), 0, []
    for (_, _, n), (_, _, _, kind) in zip(asked, streams):
        out.append(_as_kind(v[done:done + n], kind).cpu().numpy())
        done += n
    return out
