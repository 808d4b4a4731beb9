"""What a user of cafe_b200 has it do, as cases that can be timed and whose outputs can be compared.

Five kinds of work, each through the entry points that a training or serving program calls:

  train     one step of all sketch fields of a model: pooled = SKEmbeddingGroup(ids), pooled.backward(gradient), which
            runs lookup, importance, sketch insert, migration and SGD in place
  eval      the same lookup alone, without gradients (the test loop of a training script, or serving)
  bags      the drop-in module field by field, as the reference's model drives it: forward of every SKEmbeddingBag, one
            backward, insert_grad and the update of every field
  onestage  a step of SigmodSKEmbeddingBag, the one-stage sketch of the artifact tree
  interact  the dot interaction of DLRM, forward and backward

Shapes: the fields of the click-log datasets and of the micro-benchmark in cafe_b200.synthetic, with the compress and
hash rates, dimensions and batches that this repository's tests and bench.py use; "mixed" is a generic set of fields.
The ids of a field are bounded Zipf(s) ranks, scattered over the field by a seeded bijection; gradients are
N(0, 0.01^2).  A sketch has been fed some steps of its own before the first pass, so that passes meet a warm one, and
every pass takes the next of a set of batches.
"""
import math

import torch
from torch.nn.parameter import Parameter

import cafe_b200
from cafe_b200 import sizing, synthetic
from cafe_b200.dlrm_harness import fused_dot_interaction

MOST_LOOKUPS = 26 * 65536
ALPHA = 1.0000005


def _cards(case):
    shape, n = case["shape"], case["fields"]
    if shape == "mixed":   # n cardinalities from 1e3 to 1e7, evenly over the logarithm, in no order
        lo, hi = math.log(1e3), math.log(1e7)
        return [int(math.exp(lo + (hi - lo) * ((k * 7) % n + 0.5) / n)) for k in range(n)]
    cards = {"kaggle": synthetic.KAGGLE_CARDS, "terabyte": synthetic.TERABYTE_CARDS, "avazu": synthetic.AVAZU_CARDS,
             "micro": synthetic.MICRO_CARDS}[shape]
    cards = [c for c in cards if sizing.is_sketch_field(c, case["compress"])]
    return cards[:n]


def listed():
    def train(name, shape, fields, dim, batch, compress, hash_rate, zipf, ids):
        return dict(name=name, kind="train", shape=shape, fields=fields, dim=dim, batch=batch, compress=compress, hash_rate=hash_rate,
                    zipf=zipf, ids=ids)
    return [
        # the reference's own Kaggle run: mini-batch 128, dimension 16; latency and launches are all there is
        train("train_kaggle_d16_b128", "kaggle", 26, 16, 128, 0.001, 0.3, 1.1, "int64"),
        # its Terabyte run
        train("train_terabyte_d128_b2048", "terabyte", 26, 128, 2048, 0.001, 0.3, 1.1, "int64"),
        # its Avazu run: few fields, a hot table that is large for the lookups
        train("train_avazu_d16_b4096", "avazu", 9, 16, 4096, 0.1, 0.7, 1.0, "int64"),
        # an odd one: ragged batch, 32-bit ids, a middling dimension
        train("train_mixed_d64_b777", "mixed", 11, 64, 777, 0.01, 0.5, 1.05, "int32"),
        # the micro-benchmark of bench.py: the largest step, bound by the rows' traffic
        train("train_micro_d128_b65536", "micro", 26, 128, 65536, 0.001, 0.3, 1.05, "int64"),
        # large batches into a small sketch: long chains of lookups per bucket
        train("train_terabyte_tiny_b65536", "terabyte", 26, 128, 65536, 0.0001, 0.2, 1.1, "int64"),
        # serving a handful of requests
        dict(name="eval_kaggle_d16_b16", kind="eval", shape="kaggle", fields=26, dim=16, batch=16, compress=0.001, hash_rate=0.3,
             zipf=1.1, ids="int64"),
        # the test loop's batches
        dict(name="eval_terabyte_d128_b16384", kind="eval", shape="terabyte", fields=26, dim=128, batch=16384, compress=0.001,
             hash_rate=0.3, zipf=1.1, ids="int64"),
        # the drop-in module where a model holds one per field
        dict(name="bags_mixed_d64_b2048", kind="bags", shape="mixed", fields=4, dim=64, batch=2048, compress=0.01, hash_rate=0.3,
             zipf=1.05, ids="int64"),
        # the artifact tree's sketch
        dict(name="onestage_d32_b4096", kind="onestage", card=1_000_000, hot=20_000, hash_rows=5_000, dim=32, batch=4096,
             threshold=4, zipf=1.05, ids="int64"),
        # the interaction at the Terabyte run's shape, and at the largest batch with a smaller dimension
        dict(name="interact_f26_d128_b2048", kind="interact", fields=26, dim=128, batch=2048),
        dict(name="interact_f26_d64_b65536", kind="interact", fields=26, dim=64, batch=65536),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["train"] * 5 + ["eval"] * 2 + ["bags", "onestage", "interact"])
    dim = rng.choice([16, 32, 64, 128])
    ids = rng.choice(["int64", "int64", "int32"])
    if kind == "interact":
        return dict(kind=kind, fields=rng.randint(2, 32), dim=dim, batch=_log_int(rng, 16, min(65536, 65536 * 64 * 26 // (32 * dim))))
    if kind == "onestage":
        hot = _log_int(rng, 2_000, 60_000)
        return dict(kind=kind, card=_log_int(rng, 100_000, 10_000_000), hot=hot, hash_rows=_log_int(rng, 500, 50_000), dim=dim,
                    batch=_log_int(rng, 64, 16384), threshold=rng.randint(2, 8), zipf=round(rng.uniform(1.0, 1.2), 3), ids=ids)
    shape = rng.choice(["kaggle", "terabyte", "avazu", "micro", "mixed"])
    lo, hi = {"kaggle": (5e-4, 5e-3), "terabyte": (1e-4, 1e-3), "avazu": (1e-2, 1e-1), "micro": (1e-4, 1e-3), "mixed": (2e-3, 2e-2)}[shape]
    c = dict(kind=kind, shape=shape, fields=rng.randint(2, 5) if kind == "bags" else rng.randint(3, 26), dim=dim, batch=0,
             compress=float("%.3g" % math.exp(rng.uniform(math.log(lo), math.log(hi)))), hash_rate=rng.choice([0.2, 0.3, 0.5, 0.7]),
             zipf=round(rng.uniform(1.0, 1.2), 3), ids=ids)
    cards = _cards(c)
    c["fields"] = len(cards)
    # a sketch of a reasonable size for its calls: at most 128 lookups per hot row in one step
    hot = sizing.hot_rows(sum(cards), c["compress"], c["hash_rate"], dim)
    most = min(8192 if kind == "bags" else 65536, MOST_LOOKUPS * 128 // (len(cards) * dim), MOST_LOOKUPS // len(cards), 128 * hot // len(cards))
    c["batch"] = _log_int(rng, min(1 if kind == "eval" else 32, most), most)
    return c


# ---- inputs ------------------------------------------------------------------------------------------------
def _scatter(r, n, seed):
    """A seeded bijection of [0, n) applied to r: multiply and xor-shift modulo the next power of two, again for values
    that land outside."""
    bits = max(2, (n - 1).bit_length())
    mask, half = (1 << bits) - 1, bits // 2
    a, b = (0x9E3779B1 ^ (seed * 0x632BE5AB)) & 0x7FFFFFFF | 1, (seed * 0x85EBCA6B + 0x27D4EB2F) & mask
    x, todo = r.clone(), torch.ones_like(r, dtype=torch.bool)
    while bool(todo.any()):
        v = (x * (a & mask | 1) + b) & mask
        v = v ^ (v >> half)
        v = (v * 0x5BD1E995) & mask
        v = v ^ (v >> half)
        x = torch.where(todo, v, x)
        todo = x >= n
    return x


def _ids(n, shape, s, seed, gen):
    u = torch.rand(shape, dtype=torch.float64, device="cuda", generator=gen)
    if abs(s - 1.0) < 1e-9:
        r = torch.pow(float(n + 1), u) - 1
    else:
        r = torch.pow(u * ((n + 1.0) ** (1.0 - s) - 1.0) + 1.0, 1.0 / (1.0 - s)) - 1
    return _scatter(r.floor().clamp_(0, n - 1).long(), n, seed)


def _batches(case, cards, seed, warm):
    """ids of the passes [K, F, B], ids of the warm-up [warm, F, Bw], gradients [K', B, F, D]."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)
    B, D, F = case["batch"], case["dim"], len(cards)
    K = max(6, min(64, (1 << 21) // (F * B)))
    Bw = max(B, 1024) if case["kind"] == "eval" else B
    dt = torch.int32 if case["ids"] == "int32" else torch.int64
    ids = torch.stack([_ids(n, (K, B), case["zipf"], 31 * f + 7, gen) for f, n in enumerate(cards)], dim=1).to(dt).contiguous()
    first = torch.stack([_ids(n, (warm, Bw), case["zipf"], 31 * f + 7, gen) for f, n in enumerate(cards)], dim=1).to(dt).contiguous()
    G = 2 if case["kind"] == "eval" else min(K, 6)
    grads = torch.randn(G, Bw, F, D, device="cuda", generator=gen).mul_(0.01)
    return ids, first, grads


def _warm_steps(case, lookups):
    return max(10, min(40, (1 << 20) // lookups))


class _State:
    def __init__(self, case):
        self.case, self.kind, self.turn = case, case["kind"], 0

    def next(self):
        self.turn += 1
        return (self.turn - 1) % self.ids.shape[0]


def prepare(case, seed):
    st = _State(case)
    D, B, lr = case.get("dim"), case["batch"], 0.1
    torch.manual_seed(int(seed))
    if st.kind == "interact":
        gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)
        st.x = torch.randn(B, D, device="cuda", generator=gen).requires_grad_(True)
        st.emb = torch.randn(B, case["fields"], D, device="cuda", generator=gen).mul_(0.3).requires_grad_(True)
        nv = case["fields"] + 1
        st.grad = torch.randn(B, D + nv * (nv - 1) // 2, device="cuda", generator=gen).mul_(0.01)
        return st
    if st.kind == "onestage":
        cards, case = [case["card"]], dict(case)
        hot, rows = case["hot"], case["hash_rows"]
        st.sketch = cafe_b200.SigmodSketch(hot, case["threshold"], 0.99, max_lookups=B)
        gen = torch.Generator(device="cuda").manual_seed(int(seed) + 5)
        st.high = Parameter((torch.rand(hot, D, device="cuda", generator=gen) * 2 - 1) * 0.01)
        st.bags = [cafe_b200.SigmodSKEmbeddingBag(0, hot, st.sketch, st.high, "cuda", cards[0], D, 0, rows, False, max_batch=B)]
    else:
        cards = _cards(case)
        F = len(cards)
        if st.kind == "bags":
            hot = sizing.hot_rows(sum(cards), case["compress"], case["hash_rate"], D)
            st.sketch = cafe_b200.HotSketch(hot, 1, 1, ALPHA, max_lookups=B)
            gen = torch.Generator(device="cuda").manual_seed(int(seed) + 5)
            st.high = Parameter((torch.rand(hot, D, device="cuda", generator=gen) * 2 - 1) * 0.01)
            st.bags = [cafe_b200.SKEmbeddingBag(F, hot, st.sketch, st.high, "cuda", n, D, off, sizing.hash_rows(n, case["compress"], case["hash_rate"]))
                       for n, off in zip(cards, sizing.field_offsets(cards))]
        else:
            st.group = cafe_b200.SKEmbeddingGroup(cards, D, case["compress"], case["hash_rate"], 1, 1, ALPHA, device="cuda",
                                                  max_batch=max(B, 1024) if st.kind == "eval" else B, lr=lr, seed=int(seed))
    warm = _warm_steps(case, len(cards) * B)
    st.ids, first, st.grads = _batches(case, cards, seed, warm)
    if st.kind in ("train", "eval"):
        for w in range(warm):
            st.group(first[w]).backward(st.grads[w % st.grads.shape[0]])
        if st.kind == "eval":
            st.group.eval()
            st.grads = None
    else:
        if st.kind == "bags":   # as the parts of one model's output
            st.grads = st.grads.transpose(1, 2).contiguous()
        for w in range(warm):
            _bags_step(st, first[w], st.grads[w % st.grads.shape[0]])
    return st


# ---- passes ------------------------------------------------------------------------------------------------
def _bags_step(st, ids, grad):
    outs = [bag(ids[f]) for f, bag in enumerate(st.bags)]
    if st.kind == "onestage":
        outs[0].backward(grad[:, 0, :])
    else:
        torch.autograd.backward(outs, [grad[f] for f in range(len(outs))])
    masks = [bag.insert_grad(ids[f]) for f, bag in enumerate(st.bags)]
    for bag in st.bags:
        bag.apply_update(0.1)
    return outs, masks


def run(st):
    if st.kind == "interact":
        out = fused_dot_interaction(st.x, st.emb)
        gx, ge = torch.autograd.grad(out, [st.x, st.emb], st.grad)
        return [out, gx, ge]
    k = st.next()
    if st.kind == "eval":
        with torch.no_grad():
            out = st.group(st.ids[k])
        return [out, st.group.last_rows]
    grad = st.grads[k % st.grads.shape[0]]
    if st.kind == "train":
        out = st.group(st.ids[k])
        out.backward(grad)
        return [out, st.group.last_rows, st.group.weight_high] + list(st.group.weight_hash)
    outs, masks = _bags_step(st, st.ids[k], grad)
    return outs + masks + [st.high] + [bag.weight_hash for bag in st.bags]


# ---- what a pass cannot do without ----------------------------------------------------------------------------
def _distinct(n, batch, s):
    """Expected number of distinct ids among `batch` Zipf(s) draws from n."""
    edges = [1.0]
    while edges[-1] < n + 1:
        edges.append(min(n + 1.0, max(edges[-1] + 1, edges[-1] * 1.05)))

    def cdf(x):
        return math.log(x) / math.log(n + 1) if abs(s - 1) < 1e-9 else (x ** (1 - s) - 1) / ((n + 1.0) ** (1 - s) - 1)
    tot = 0.0
    for a, b in zip(edges, edges[1:]):
        tot += (b - a) * -math.expm1(-batch * (cdf(b) - cdf(a)) / (b - a))
    return tot


def work(case):
    B, D = case["batch"], case["dim"]
    row = 4.0 * D
    if case["kind"] == "interact":
        nv = case["fields"] + 1
        pairs = nv * (nv - 1) // 2
        # forward: the vectors in, the row out; backward: the incoming row and the vectors in, their gradients out
        return {"bytes": B * (3.0 * nv * row + 2.0 * 4 * (D + pairs)), "flops": B * (2.0 * pairs * D + 4.0 * pairs * D)}
    cards = [case["card"]] if case["kind"] == "onestage" else _cards(case)
    L = B * len(cards)
    u = sum(_distinct(n, B, case["zipf"]) for n in cards)
    idb = 4 if case["ids"] == "int32" else 8
    if case["kind"] == "eval":   # id in, row and row code out; a bucket's 32 bytes and the row of every distinct id
        return {"bytes": L * (idb + row + 4) + u * (32 + row), "flops": 0}
    # id and gradient row in, pooled row and row code out; bucket (64 bytes) and row of every distinct id in and out
    return {"bytes": L * (idb + 2 * row + 4) + u * 2 * (64 + row), "flops": 4.0 * L * D}


def tolerance(case):
    # Against the same sums in 64 bits: the interaction's outputs are off by up to 1.9e-7 (largest element 2.7e-6); the
    # tables of one step by up to 1.2e-7 (1.5e-5), which the steps before the first pass have done ten to forty times.
    # Importances decide which ids are hot, so they and the row codes are the same to the bit.
    if case["kind"] == "interact":
        return {"rel": 1e-6, "max": 2e-5}
    return {"rel": 2e-6, "max": 4e-4}
