"""The work a user of this framework has it do, as cases that can be timed and compared.

Each case is one pass through a public entry point with inputs made from a seed:

* per photo: ``features.sift_gpu_u8`` (the feature worker: host image in, feature-file content out),
  ``gsift.detect`` + ``gsift.describe`` (keypoints with a state, then their descriptors),
  ``features.sift_gpu_batch_d`` (a batch of photos resident on the device);
* per flight: ``frontend.extract_and_match`` (page-locked photos in, match lists and features out);
* per pair: ``matching._ratio_match_bf`` (the coarse stage of a pair, host arrays),
  ``matching.ratio_match_bf_batch_d`` (exhaustive matching of many pairs, each distance engine) and
  ``matching.guided_from_pred_batch_d`` (prior-guided matching of many pairs);
* the learned match filter: ``match_filter.MatchFilter.predict`` + ``accept`` and ``fit``.

Photos are synthetic (seeded terrain texture plus sensor noise, as the synthetic flight's frames),
descriptors are SIFT-like uint8 rows with a share of true correspondences.
"""
import math

import numpy as np
import torch

import fieldstitch_b200 as F
from fieldstitch_b200 import match_filter, synth

CONTRAST, EDGE = 0.015, 12.0   # the reference's defaults for aerial photos
RADIUS, KC, RATIO = 40.0, 16, 0.85
N_FEAT, HID = 8, 64            # the match filter's network: 8-64-64-1


# ------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a thumbnail-sized photo: the smallest per-photo call, launches and waits count
        {"name": "photo_320x240", "kind": "photo", "h": 240, "w": 320, "nfeat": 1000},
        # an odd-sized, ragged photo (no octave width is a multiple of four)
        {"name": "photo_1321x989", "kind": "photo", "h": 989, "w": 1321, "nfeat": 4000},
        # the ordinary photo of a flight (reduced to 2640 x 1978) with the pipeline's feature cap
        {"name": "photo_2640x1978", "kind": "photo", "h": 1978, "w": 2640, "nfeat": 12000},
        # detect + describe with OpenCV's default thresholds, every keypoint described
        {"name": "detect_1320x989", "kind": "detect", "h": 989, "w": 1320, "max_kp": 8000},
        # a batch of photos resident on the device, uneven feature caps: the flight's bulk extraction
        {"name": "batch_16x2640x1978", "kind": "batch", "n": 16, "h": 1978, "w": 2640, "lo": 2000, "hi": 16000},
        # the whole front end for a strip of a flight: photos in, matches and features out
        {"name": "flight_8x12", "kind": "flight", "n": 8, "pairs": 12, "h": 1978, "w": 2640, "nfeat": 7000},
        # the coarse stage of one pair: the 1500 strongest features of each photo, host arrays
        {"name": "coarse_1500", "kind": "coarse", "na": 1500, "nb": 1500},
        # exhaustive matching of pairs without a usable prior, plain distances
        {"name": "dense_fp32_4", "kind": "dense", "prec": "fp32", "n": 4, "lo": 5001, "hi": 8999},
        # dense matching of many large pairs on the tensor cores
        {"name": "dense_bf16_16", "kind": "dense", "prec": "bf16", "n": 16, "lo": 16384, "hi": 16384},
        # the same with 8-bit operands and uneven pairs
        {"name": "dense_fp8_24", "kind": "dense", "prec": "fp8", "n": 24, "lo": 2000, "hi": 16000},
        # prior-guided matching of a flight's pairs, uneven keypoint counts
        {"name": "guided_64", "kind": "guided", "n": 64, "lo": 2000, "hi": 16000},
        # the learned filter: training on the correspondences of a flight's first pairs, and scoring
        {"name": "filter_390k", "kind": "filter", "n": 390001, "epochs": 4, "batch": 8192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["photo", "photo", "photo", "detect", "batch", "flight", "coarse", "dense", "dense", "dense",
                       "guided", "filter"])
    if kind in ("photo", "detect"):
        h = _log(rng, 200, 1978)
        w = min(2640, max(200, int(h * rng.uniform(0.75, 1.5))))
        if kind == "photo":
            return {"kind": kind, "h": h, "w": w, "nfeat": _log(rng, 500, 16000)}
        return {"kind": kind, "h": min(h, 1400), "w": min(w, 1900), "max_kp": _log(rng, 500, 12000)}
    if kind == "batch":
        h = _log(rng, 480, 1978)
        return {"kind": kind, "n": rng.randint(2, 14), "h": h, "w": int(h * rng.uniform(1.0, 1.33)),
                "lo": rng.randint(500, 4000), "hi": rng.randint(4001, 12000)}
    if kind == "flight":
        n = rng.randint(2, 7)
        h = _log(rng, 480, 1978)
        return {"kind": kind, "n": n, "pairs": rng.randint(1, n * (n - 1) // 2), "h": h,
                "w": int(h * rng.uniform(1.0, 1.33)), "nfeat": _log(rng, 500, 8000)}
    if kind == "coarse":
        return {"kind": kind, "na": _log(rng, 200, 4000), "nb": _log(rng, 200, 4000)}
    if kind == "dense":
        prec = rng.choice(["fp32", "bf16", "fp8"])
        n = rng.randint(1, 4) if prec == "fp32" else _log(rng, 1, 20)
        lo = _log(rng, 300, 6000)
        return {"kind": kind, "prec": prec, "n": n, "lo": lo, "hi": rng.randint(lo + 1, 9000 if prec == "fp32" else 14000)}
    if kind == "guided":
        lo = _log(rng, 500, 6000)
        return {"kind": kind, "n": _log(rng, 1, 60), "lo": lo, "hi": rng.randint(lo + 1, 14000)}
    return {"kind": kind, "n": _log(rng, 20000, 390000), "epochs": rng.randint(1, 4), "batch": rng.choice([2048, 4096, 8192])}


# ------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _sizes(case, k=1):
    """`n` rows of k uneven sizes in [lo, hi]; the same for every seed, so that outputs keep their shapes."""
    r = np.random.default_rng([case["n"], case["lo"], case["hi"]])
    return r.integers(case["lo"], case["hi"] + 1, (case["n"], k))


def _rows(a, n):
    """`a` with n rows (zeros after its own): lists whose length depends on the data."""
    if len(a) == n:
        return a
    if isinstance(a, torch.Tensor):
        out = torch.zeros((n,) + tuple(a.shape[1:]), dtype=a.dtype, device=a.device)
    else:
        out = np.zeros((n,) + a.shape[1:], a.dtype)
    out[:len(a)] = a
    return out


def _photo(h, w, seed):
    """uint8 (h, w) CUDA image: seeded terrain texture plus sensor noise (sigma 2)."""
    t = synth.flight_terrain(seed, h, w).to(torch.float32)
    t += 2.0 * torch.randn(t.shape, generator=_gen(seed + 1), device="cuda")
    return torch.clamp(torch.round(t), 0, 255).to(torch.uint8)


def _pairs_of(n, m):
    """The first m pairs of n frames in flight order: neighbours first, then the next ones."""
    every = [(i, i + d) for d in range(1, n) for i in range(n - d)]
    return every[:m]


def _correspondences(n, seed):
    """(features (n, 8) float32, labels (n,) float32) CUDA with the match filter's distributions:
    true candidates have a smaller ratio, distance, angle difference and residual."""
    g = _gen(seed)

    def normal():
        return torch.randn(n, generator=g, device="cuda")

    def uniform():
        return torch.rand(n, generator=g, device="cuda")

    true = uniform() < 0.55
    a, b = normal().abs(), uniform()
    f = torch.stack([
        torch.where(true, 0.35 + 0.2 * a, 0.75 + 0.25 * b).clamp(0, 1.0),          # ratio
        torch.where(true, 0.25 + 0.1 * a, 0.55 + 0.15 * a),                        # best distance
        torch.where(true, 0.15 * normal(), 0.9 * normal()),                        # log2 scale ratio
        torch.where(true, 0.05 * normal(), 2.0 * uniform() - 1.0).clamp(-1, 1),    # angle difference
        torch.where(true, 0.25 * a, b.sqrt()).clamp(0, 1),                         # prior residual
        0.005 + 0.02 * normal().abs(), 0.005 + 0.02 * normal().abs(),              # responses
        torch.floor(-torch.log2(uniform().clamp_min(1e-3)) * 0.5)], 1)             # octave
    label = torch.where(uniform() < 0.03, ~true, true).to(torch.float32)
    return f.to(torch.float32).contiguous(), label


def _start_params(seed):
    """A freshly initialised network, with the input normalisation of the distribution above."""
    r = np.random.default_rng(seed)
    p = [r.normal(0, math.sqrt(2 / N_FEAT), HID * N_FEAT), np.zeros(HID), r.normal(0, math.sqrt(2 / HID), HID * HID),
         np.zeros(HID), r.normal(0, math.sqrt(1 / HID), HID), np.zeros(1),
         np.array([0.67, 0.5, 0.0, 0.0, 0.42, 0.021, 0.021, 0.36]), np.array([0.25, 0.19, 0.62, 0.4, 0.28, 0.012, 0.012, 0.77])]
    return np.concatenate(p).astype(np.float32)


def _filter_sets(case, seed):
    feat, label = _correspondences(case["n"], seed)
    g = _gen(seed + 5)
    nb = max(1000, case["n"] // 2)
    t1 = torch.randint(0, nb, (case["n"],), generator=g, device="cuda", dtype=torch.int32)
    t1[torch.rand(case["n"], generator=g, device="cuda") < 0.05] = -1
    b1 = torch.round((feat[:, 1] * 512.0) ** 2)
    b12 = torch.stack([b1, torch.round(b1 / (feat[:, 0] ** 2).clamp_min(1e-3))], 1).contiguous()
    return feat, label, t1, b12, nb


def prepare(case, seed):
    k = case["kind"]
    if k in ("photo", "detect"):
        return {"case": case, "img": _photo(case["h"], case["w"], seed).cpu().numpy()}
    if k == "batch":
        n, h, w = case["n"], case["h"], case["w"]
        caps = [int(v) for v in _sizes(case)[:, 0]]
        img = torch.stack([_photo(h, w, 1000 * seed + i) for i in range(n)])
        return {"case": case, "img": img, "caps": caps,
                "xy": torch.zeros((n, max(caps), 2), dtype=torch.float32, device="cuda"),
                "u8": torch.zeros((n, max(caps), 128), dtype=torch.uint8, device="cuda"),
                "rs": torch.zeros((n, max(caps)), dtype=torch.float32, device="cuda")}
    if k == "flight":
        n, h, w = case["n"], case["h"], case["w"]
        # two flight lines of frames, 80 % forward and 70 % side overlap
        poses = synth.lawnmower(seed, lines=2, per_line=(n + 1) // 2, W=w, H=h, margin=0.2 * max(h, w))[:n]
        th, tw = (int(poses[:, 1].max() + 0.8 * max(h, w)), int(poses[:, 0].max() + 0.8 * max(h, w)))
        frames = synth.render_frames(synth.flight_terrain(seed, th, tw), poses, w, h, seed=seed)
        pairs = _pairs_of(n, case["pairs"])
        off = np.random.default_rng(seed).normal(0.0, 15.0, (len(pairs), case["nfeat"], 2)).astype(np.float32)
        return {"case": case, "frames": [f.cpu().pin_memory().numpy() for f in frames], "pairs": pairs,
                "priors": [synth.frame_homography(poses[i], poses[j], w, h) for i, j in pairs], "off": list(off),
                "qt": np.zeros((len(pairs), 2, case["nfeat"]), np.int64)}
    if k == "coarse":
        a, b, _ = synth.synth_descriptors_device(case["na"], case["nb"], seed)
        return {"case": case, "a": a.cpu().numpy(), "b": b.cpu().numpy()}
    if k == "dense":
        s = _sizes(case, 2)
        ab = [synth.synth_descriptors_device(int(na), int(nb), 1000 * seed + i)[:2] for i, (na, nb) in enumerate(s)]
        m = int(s[:, 0].max())
        return {"case": case, "a": [a for a, _ in ab], "b": [b for _, b in ab],
                "q": torch.zeros((len(ab), m), dtype=torch.int64, device="cuda"),
                "t": torch.zeros((len(ab), m), dtype=torch.int64, device="cuda")}
    if k == "guided":
        w, h = 2640.0, 1978.0
        wh = torch.tensor([w, h], dtype=torch.float64, device="cuda")
        s = _sizes(case, 2)
        probs = []
        for i, (na, nb) in enumerate(s):
            g = _gen(1000 * seed + i)
            a, b, truth = synth.synth_descriptors_device(int(na), int(nb), 1000 * seed + i)
            bxy = torch.rand((int(nb), 2), generator=g, dtype=torch.float64, device="cuda") * wh
            pred = torch.rand((int(na), 2), generator=g, dtype=torch.float64, device="cuda") * wh
            j = torch.nonzero(truth >= 0)[:, 0]
            pred[truth[j]] = bxy[j] + 15.0 * torch.randn((len(j), 2), generator=g, dtype=torch.float64, device="cuda")
            probs.append((pred.contiguous(), a, bxy.contiguous(), b, (w, h)))
        m = int(s[:, 0].max())
        q = torch.zeros((len(s), m), dtype=torch.int64, device="cuda")
        t = torch.zeros((len(s), m), dtype=torch.int64, device="cuda")
        return {"case": case, "probs": probs, "q": q, "t": t, "out": [(q[i], t[i]) for i in range(len(s))]}
    feat, label, t1, b12, nb = _filter_sets(case, seed)
    return {"case": case, "feat": feat, "label": label, "t1": t1, "b12": b12, "nb": nb, "params": _start_params(seed),
            "seed": int(seed) & 0xffff}


# ------------------------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "photo":
        res = F.features.sift_gpu_u8(state["img"], case["nfeat"], CONTRAST, EDGE)
        return [_rows(a, case["nfeat"]) for a in res], len(res[0])
    if k == "detect":
        kps, st = F.gsift.detect(state["img"], max_kp=case["max_kp"], contrast=0.04, edge=10.0)
        desc = F.gsift.describe(st, kps, np.arange(len(kps["x"])))
        st.close()
        return {n: _rows(a, case["max_kp"]) for n, a in kps.items()}, _rows(desc, case["max_kp"]), len(desc)
    if k == "batch":
        n = case["n"]
        counts = F.features.sift_gpu_batch_d([state["img"][i] for i in range(n)], state["caps"],
                                             [state["xy"][i] for i in range(n)], [state["u8"][i] for i in range(n)],
                                             [state["rs"][i] for i in range(n)])
        return np.array(counts), state["xy"], state["u8"], state["rs"]
    if k == "flight":
        matches, feats = F.frontend.extract_and_match(state["frames"], case["nfeat"], state["pairs"], state["priors"],
                                                      RADIUS, KC, RATIO, offsets=state["off"], return_features=True)
        for p, (q, t) in enumerate(matches):
            state["qt"][p, 0, :len(q)] = q
            state["qt"][p, 1, :len(t)] = t
        return (np.array([len(q) for q, _ in matches]), state["qt"],
                [[_rows(a, case["nfeat"]) for a in f] for f in feats])
    if k == "coarse":
        q, t = F.matching._ratio_match_bf(state["a"], state["b"], RATIO)
        return len(q), _rows(q, case["na"]), _rows(t, case["na"])
    if k == "dense":
        res = F.matching.ratio_match_bf_batch_d(state["a"], state["b"], 0.8, precision=case["prec"],
                                                out=[(state["q"][i], state["t"][i]) for i in range(case["n"])])
        return np.array([len(q) for q, _ in res]), state["q"], state["t"]
    if k == "guided":
        res = F.matching.guided_from_pred_batch_d(state["probs"], RADIUS, KC, RATIO, out=state["out"])
        return np.array([len(q) for q, _ in res]), state["q"], state["t"]
    net = match_filter.MatchFilter(state["params"])
    losses = net.fit(state["feat"], state["label"], epochs=case["epochs"], batch=case["batch"], seed=state["seed"])
    # scores by the network that the program started with: what a stored network gives
    prob = match_filter.MatchFilter(state["params"]).predict(state["feat"])
    q, t = match_filter.accept(state["t1"], state["b12"], state["nb"], prob)
    return losses, net.params, prob, len(q), _rows(q, case["n"]), _rows(t, case["n"])


# ------------------------------------------------------------------------------------ work
def _octave_pixels(h, w):
    r, c, tot = 2 * h, 2 * w, 0
    while min(r, c) >= 14:
        tot += r * c
        r, c = (r + 1) // 2, (c + 1) // 2
    return tot


def _photo_work(h, w, nfeat, row):
    """One photo: the image in, its features out (row bytes each); the separable blurs' multiply-adds
    (11 taps for the base, 11 + 13 + 17 + 21 + 27 per octave pixel, both axes)."""
    return h * w + nfeat * row, 2 * 2 * (11 * 4 * h * w + 89 * _octave_pixels(h, w))


def work(case):
    k = case["kind"]
    mid = (case.get("lo", 0) + case.get("hi", 0)) // 2
    if k == "photo":
        b, f = _photo_work(case["h"], case["w"], case["nfeat"], 8 + 4 + 128)
    elif k == "detect":
        b, f = _photo_work(case["h"], case["w"], case["max_kp"], 7 * 4 + 512)
    elif k == "batch":
        b, f = (case["n"] * v for v in _photo_work(case["h"], case["w"], mid, 8 + 4 + 128))
    elif k == "flight":
        b, f = (case["n"] * v for v in _photo_work(case["h"], case["w"], case["nfeat"], 8 + 4 + 128))
        b += case["pairs"] * case["nfeat"] * 24
        f += case["pairs"] * case["nfeat"] * KC * 256
    elif k == "coarse":
        b, f = 128 * (case["na"] + case["nb"]) + 16 * case["na"], 256.0 * case["na"] * case["nb"]
    elif k == "dense":
        b, f = case["n"] * (128 * 2 * mid + 16 * mid), case["n"] * 256.0 * mid * mid
    elif k == "guided":
        b, f = case["n"] * mid * (16 + 128 + 16 + 128 + 16), case["n"] * mid * KC * 256.0
    else:
        macs = HID * N_FEAT + HID * HID + HID
        b = case["n"] * (4 * N_FEAT + 4) * case["epochs"] + case["n"] * (4 * N_FEAT + 12 + 4 + 16)
        f = 2.0 * macs * case["n"] * (3 * case["epochs"] + 1)
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------------------------------ 64 bits
def _unpack(p):
    o, out = 0, []
    for n, shape in ((HID * N_FEAT, (HID, N_FEAT)), (HID, (HID,)), (HID * HID, (HID, HID)), (HID, (HID,)), (HID, (HID,)),
                     (1, (1,)), (N_FEAT, (N_FEAT,)), (N_FEAT, (N_FEAT,))):
        out.append(p[o:o + n].reshape(shape))
        o += n
    return out


def _net(p, x):
    w1, b1, w2, b2, w3, b3, mu, sig = _unpack(p)
    h = torch.relu(((x - mu) / sig) @ w1.T + b1)
    return torch.relu(h @ w2.T + b2) @ w3 + b3


def _shuffle(n, epoch, seed):
    """The epoch's sample order: a stable sort by a 32-bit hash of (seed, epoch, sample)."""
    m = 0xffffffff
    i = torch.arange(n, device="cuda", dtype=torch.int64)

    def mul(a, c):   # 32-bit product (the low half only, in two parts)
        return ((a * (c & 0xffff)) + (((a * (c >> 16)) & 0xffff) << 16)) & m

    h = mul(i, 0x85EBCA6B) ^ ((int(seed) ^ (0x9E3779B9 * (epoch + 1))) & m)
    h ^= h >> 16
    h = mul(h, 0x7FEB352D)
    h ^= h >> 15
    h = mul(h, 0x846CA68B)
    h ^= h >> 16
    return torch.sort(h, stable=True)[1]


def exact(case, seed):
    """The filter's training and scores in 64 bits. The other cases return whole numbers, or
    keypoints whose number and order 64-bit arithmetic would change."""
    if case["kind"] != "filter":
        return None
    feat, label, _, _, _ = _filter_sets(case, seed)
    x, y = feat.double(), label.double()
    start = torch.from_numpy(_start_params(seed)).cuda().double()
    p = start.clone()
    n_train = p.numel() - 2 * N_FEAT
    m, v = torch.zeros(n_train, device="cuda", dtype=torch.float64), torch.zeros(n_train, device="cuda", dtype=torch.float64)
    n = case["n"]
    batch = min(n, max(128, case["batch"] // 128 * 128))
    steps, losses, t = max(1, n // batch), [], 0
    for e in range(case["epochs"]):
        order = _shuffle(n, e, int(seed) & 0xffff)
        total = 0.0
        for s in range(steps):
            idx = order[s * batch:(s + 1) * batch]
            q = p.detach().requires_grad_(True)
            loss = torch.nn.functional.binary_cross_entropy_with_logits(_net(q, x[idx]), y[idx])
            g = torch.autograd.grad(loss, q)[0][:n_train]
            t += 1
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p = p.detach()
            p[:n_train] -= 2e-3 * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
            total += float(loss.detach())
        losses.append(total / steps)
    prob = torch.sigmoid(_net(start, x))
    return np.array(losses), p, prob, None, None, None
