"""The work that users of this package have it do, as cases that can be timed.

    position   Engine.perft_position: one GPU perft of one position
    launch     Engine.perft_launch: one depth through the host driver (splits
               above the launch depth), no tables
    iterate    Engine.perft on a FEN: the command line's per-depth loop
    tables     a whole run with transposition tables, engine and all (a kept
               engine would answer a repeated position from its tables)
    batch      Engine.perft_batch: many roots at one depth
    label      Engine.perft_batch at depths 1..4: the scheduler network's labels
    planned    Engine.perft_batch_planned: roots at mixed depths, sizes
               predicted by a trained network
    predict    Engine.mlp_predict: size predictions of a batch of positions
    train      Engine.mlp_train: the network trained on labelled positions

Positions are playouts of uniformly random legal moves, as in the benchmark
and the tests; plies says how far into the game they are.  An engine is kept
by the user's program between calls, so prepare() makes it.
"""
import numpy as np
import torch

import perft_gpu_2026_b200 as pg

IN, H, OUT = 781, 256, 4
LR = 1e-3


def listed():
    return [
        # a tool that asks for one small perft: latency and launches
        {"name": "position d4", "kind": "position", "depth": 4, "plies": 20, "strict": False},
        # a middle-game position at a usual checking depth, exact counting convention
        {"name": "position d6 strict", "kind": "position", "depth": 6, "plies": 14, "strict": True},
        # the benchmark's shape: an opening position, perft 7
        {"name": "position d7", "kind": "position", "depth": 7, "plies": 4, "strict": False},
        # the largest run without tables: perft 8 through the host driver
        {"name": "launch d8", "kind": "launch", "depth": 8, "plies": 4, "strict": False},
        # the command line without tables: every depth up to 6
        {"name": "iterate d6", "kind": "iterate", "depth": 6, "plies": 8, "strict": False},
        # the command line with tables, start to end
        {"name": "tables d9", "kind": "tables", "depth": 9, "plies": 2, "device_mb": 8192},
        # a small suite of positions (an EPD file) at a shallow depth
        {"name": "batch 200 d4", "kind": "batch", "n": 200, "depth": 4, "lo": 6, "hi": 40},
        # thousands of uneven roots at once
        {"name": "batch 4096 d5", "kind": "batch", "n": 4096, "depth": 5, "lo": 6, "hi": 40},
        # labels for the scheduler network
        {"name": "label 20000", "kind": "label", "n": 20000, "lo": 0, "hi": 60},
        # roots at mixed depths through the learned planner
        {"name": "planned 1000", "kind": "planned", "n": 1000, "dlo": 3, "dhi": 6, "lo": 0, "hi": 60},
        # size predictions for one batch
        {"name": "predict 4096", "kind": "predict", "n": 4096, "lo": 0, "hi": 60},
        # training of the scheduler network
        {"name": "train 32768", "kind": "train", "n": 32768, "batch": 4096, "epochs": 1, "lo": 0, "hi": 60},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["position", "position", "batch", "batch", "launch", "iterate", "tables", "label", "planned",
                       "predict", "train"])
    lo = rng.randint(0, 12)
    span = {"lo": lo, "hi": lo + rng.randint(8, 48)}
    if kind == "position":
        d = rng.randint(3, 7)
        return {"kind": kind, "depth": d, "plies": rng.randint(2, 6 if d == 7 else 40), "strict": rng.random() < 0.3}
    if kind == "launch":
        return {"kind": kind, "depth": rng.randint(5, 8), "plies": rng.randint(2, 4), "strict": rng.random() < 0.3}
    if kind == "iterate":
        return {"kind": kind, "depth": rng.randint(3, 6), "plies": rng.randint(2, 30), "strict": rng.random() < 0.3}
    if kind == "tables":
        return {"kind": kind, "depth": rng.randint(6, 8), "plies": rng.randint(0, 8), "device_mb": rng.randint(2048, 8192)}
    if kind == "batch":
        d = rng.randint(1, 5)
        return {"kind": kind, "n": _log(rng, 10, (1 << 17) >> (4 * max(d - 3, 0))), "depth": d, **span}
    if kind == "label":
        return {"kind": kind, "n": _log(rng, 1000, 40000), **span}
    if kind == "planned":
        dlo = rng.randint(2, 5)
        return {"kind": kind, "n": _log(rng, 20, 1000), "dlo": dlo, "dhi": dlo + rng.randint(0, 1), **span}
    if kind == "predict":
        return {"kind": kind, "n": _log(rng, 10, 65536), **span}
    return {"kind": kind, "n": rng.randint(4096, 40000), "batch": 64 * _log(rng, 4, 64), "epochs": 1, **span}


def _positions(n, seed, lo, hi):
    """n playout positions with a legal move, as one packed array."""
    out, k = [], 0
    while len(out) < n:
        more = pg.random_playouts(seed * 64 + k, n + n // 16 + 8, lo, hi)
        out += [p for p in more if pg.count_moves(p, True) > 0]
        k += 1
    return pg.pack_positions(out[:n])


def _params(seed):
    """The network's parameters (He-uniform; biases near the mean targets), in the library's flat layout."""
    r = np.random.default_rng(seed)

    def uni(lim, *shape):
        return r.uniform(-lim, lim, size=shape).astype(np.float32).ravel()

    return np.concatenate([uni((6 / 35) ** 0.5, IN, H), uni(0.1, H), uni((6 / H) ** 0.5, H, H), uni(0.1, H),
                           uni((3 / H) ** 0.5, H, OUT), np.array([4.5, 9, 13.5, 18], dtype=np.float32)])


def _labels(eng, pos):
    return np.log2(1.0 + np.array([eng.perft_batch(pos, d) for d in (1, 2, 3, 4)], dtype=np.float64).T).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("position", "launch", "iterate", "tables"):
        pos = _positions(1, seed, case["plies"], case["plies"])[0]
        s = {"case": case, "pos": pos, "fen": pg.to_fen(pos)}
        if kind != "tables":
            s["eng"] = pg.Engine(device=0, use_tt=False, strict=case["strict"])
        return s
    s = {"case": case, "eng": pg.Engine(device=0, use_tt=False)}
    s["pos"] = _positions(case["n"], seed, case["lo"], case["hi"])
    if kind == "planned":
        # the network as the scheduler makes it: labelled playouts, a few epochs
        r = np.random.default_rng(seed)
        s["depths"] = r.integers(case["dlo"], case["dhi"] + 1, size=case["n"]).astype(np.intc)
        train = _positions(16384, seed + 1, 0, 60)
        y = _labels(s["eng"], train)
        s["eng"].mlp_init(seed=1, out_bias=list(y.mean(0)))
        s["eng"].mlp_train(train, y, epochs=40, batch=2048, lr=2e-3)
    if kind in ("predict", "train"):
        s["params"] = _params(seed)
        s["eng"].mlp_init(seed=1)
        s["eng"].mlp_set_params(s["params"])
    if kind == "train":
        s["targets"] = _labels(s["eng"], s["pos"])
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "position":
        return s["eng"].perft_position(s["pos"], case["depth"])
    if kind == "launch":
        return s["eng"].perft_launch(s["pos"], case["depth"])[0]
    if kind == "iterate":
        return [n for n, _ in s["eng"].perft(s["fen"], case["depth"])]
    if kind == "tables":
        with pg.Engine(device=0, use_tt=True, arena_bytes=8 << 30, device_tt_mb=case["device_mb"],
                       host_tt_mb=64) as eng:
            return [n for n, _ in eng.perft(s["fen"], case["depth"])]
    if kind == "batch":
        return np.array(s["eng"].perft_batch(s["pos"], case["depth"]), dtype=np.int64)
    if kind == "label":
        return [np.array(s["eng"].perft_batch(s["pos"], d), dtype=np.int64) for d in (1, 2, 3, 4)]
    if kind == "planned":
        return np.array(s["eng"].perft_batch_planned(s["pos"], s["depths"])[0], dtype=np.int64)
    if kind == "predict":
        return s["eng"].mlp_predict(s["pos"])
    # a training run from the given weights
    s["eng"].mlp_set_params(s["params"])
    loss = s["eng"].mlp_train(s["pos"], s["targets"], epochs=case["epochs"], batch=case["batch"], lr=LR)
    return {"loss": loss, "params": s["eng"].mlp_params()}


def work(case):
    """Counting a position's moves is at least one operation per move; a
    position has about 30, and the counted positions are those one ply above
    the leaves.  A root is 40 bytes, a count 8."""
    kind = case["kind"]
    if kind in ("position", "launch", "tables"):
        return {"bytes": 48, "flops": 30.0 ** case["depth"]}
    if kind == "iterate":
        return {"bytes": 40 + 8 * case["depth"], "flops": sum(30.0 ** d for d in range(1, case["depth"] + 1))}
    n = case["n"]
    if kind == "batch":
        return {"bytes": 48 * n, "flops": n * 30.0 ** case["depth"]}
    if kind == "label":
        return {"bytes": 72 * n, "flops": n * sum(30.0 ** d for d in (1, 2, 3, 4))}
    if kind == "planned":
        return {"bytes": 48 * n, "flops": n * 30.0 ** (0.5 * (case["dlo"] + case["dhi"]))}
    # layer 1 adds one row per active input (about 30 of 781)
    forward = 30 * H + 2 * H * H + 2 * H * OUT
    weights = IN * H + H + H * H + H + H * OUT + OUT
    if kind == "predict":
        return {"bytes": 56 * n + 2 * weights, "flops": float(n * forward)}
    return {"bytes": case["epochs"] * 56 * n + 16 * weights, "flops": float(case["epochs"] * n * 3 * forward)}


# ---------------------------------------------------------------- the network in 64 bits
def _inputs(pos):
    """The 781 binary inputs of each position as a float64 matrix."""
    raw = np.frombuffer(bytes(pos), dtype=np.uint8).reshape(len(pos), 40)
    bits = np.unpackbits(raw[:, :32], axis=1, bitorder="little").reshape(len(pos), 4, 64)
    black, piece = bits[:, 0], bits[:, 1] + 2 * bits[:, 2] + 4 * bits[:, 3]
    state, color = raw[:, 32].astype(int), raw[:, 33]
    x = np.zeros((len(pos), IN))
    i, sq = np.nonzero(piece)
    x[i, (black[i, sq].astype(int) * 6 + piece[i, sq] - 1) * 64 + sq] = 1
    x[color == 0, 768] = 1
    for c in range(4):
        x[(state >> c) & 1 == 1, 769 + c] = 1
    ep = state >> 4
    x[ep > 0, 773 + ep[ep > 0] - 1] = 1
    return torch.from_numpy(x).cuda()


_SIZES = [(IN, H), (H,), (H, H), (H,), (H, OUT), (OUT,)]


def _split(p):
    out, o = [], 0
    for shape in _SIZES:
        n = int(np.prod(shape))
        out.append(p[o:o + n].view(*shape))
        o += n
    return out


def _forward(p, x):
    w1, b1, w2, b2, w3, b3 = _split(p)
    w1, w2, w3 = (w.bfloat16().double() for w in (w1, w2, w3))  # the weights are held in BF16
    h1 = torch.relu(x @ w1 + b1)
    h2 = torch.relu(h1 @ w2 + b2)
    return h1, h2, h2 @ w3 + b3, (w1, w2, w3)


def exact(case, seed):
    kind = case["kind"]
    if kind == "predict":
        x = _inputs(_positions(case["n"], seed, case["lo"], case["hi"]))
        return _forward(torch.from_numpy(_params(seed)).cuda().double(), x)[2]
    if kind != "train":
        return None
    s = prepare(case, seed)
    x, t = _inputs(s["pos"]), torch.from_numpy(s["targets"]).cuda().double()
    p = torch.from_numpy(s["params"]).cuda().double()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    n, batch, step, state, losses = case["n"], case["batch"], 0, 7, []
    order = list(range(n))
    for _ in range(case["epochs"]):
        losses = []
        for i in range(n - 1, 0, -1):
            r, state = pg.splitmix64(state)
            j = (r * (i + 1)) >> 64
            order[i], order[j] = order[j], order[i]
        at = torch.tensor(order, device="cuda")
        for b in range(0, n - batch + 1, batch):
            xb, tb = x[at[b:b + batch]], t[at[b:b + batch]]
            h1, h2, y, (w1, w2, w3) = _forward(p, xb)
            d = y - tb
            losses.append(float((d * d).mean()))
            dy = 2 * d / (batch * OUT)
            d2 = (dy @ w3.T) * (h2 > 0)
            d1 = (d2 @ w2.T) * (h1 > 0)
            g = torch.cat([q.reshape(-1) for q in (xb.T @ d1, d1.sum(0), h1.T @ d2, d2.sum(0), h2.T @ dy, dy.sum(0))])
            step += 1
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p = p - LR * (m / (1 - 0.9 ** step)) / ((v / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return {"loss": sum(losses) / len(losses), "params": p}
