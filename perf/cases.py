"""What a user of this framework has it do, as cases that can be timed and compared.

A program holds one context (ring degree 2^16, twelve levels) with its keys, and one HEMMer per schedule it uses; switching
keys, masks and encoded weights are made on first use and kept.  A case is one pass of such a program from its operands to its
results, through the package's public calls.  Ciphertext results are returned as int64 tensors over the device memory that
holds their residues (all below 2^60).

Kinds of cases (sizes are those of the encoder-layer workload of `layer.py`, its parts, and the primitive sweep of `bench.py`):

  primitive   one evaluator call on a batch of ciphertexts with uniform residues: rotate | mult | rescale | ntt | intt
  product     encrypted tile x encrypted tile, `pairs` independent products at once; transpose: the operand that is transposed
              first ("right": Q K^T, "left": X^T dY); schedule 0 is the library's default, 2 the one `bench.py` times
  projection  encrypted activations x plaintext weights: k_tiles x n_tiles tiles of 128, shifted copies made once and reused
  scores      the score assembly of the Gaussian-kernel attention
  encrypt     host matrices -> ciphertexts;   decrypt: ciphertexts -> host values
  layer       all matmuls of one BERT-base encoder layer, forward and LoRA backward; end_to_end: host matrices in and out
"""
from __future__ import annotations

import importlib

import numpy as np
import torch

PKG = "encryption-friendly_llm_architecture_b200"
N, LEVELS, SPECIAL, ALPHA = 1 << 16, 12, 3, 4   # ring degree, top level, special primes, limbs of a key-switch digit
D = 128                                         # tile side
TARGET = 4                                      # level of a product's result

_held = {}


def listed():
    return [
        # the smallest call: one rotation of one fresh ciphertext (the layers around the products are made of these)
        {"name": "rotate_one", "kind": "primitive", "op": "rotate", "level": 12, "batch": 1, "step": 1},
        # the primitive sweep: 256 independent ciphertexts multiplied (tensor, relinearise, rescale)
        {"name": "mult_256", "kind": "primitive", "op": "mult", "level": 8, "batch": 256, "step": 0},
        # a single encrypted product, one tile per ciphertext, in the library's default schedule
        {"name": "product_default", "kind": "product", "pairs": 1, "tiles": 1, "schedule": 0, "transpose": ""},
        # one two-tile product in the fast schedule
        {"name": "product_one", "kind": "product", "pairs": 1, "tiles": 2, "schedule": 2, "transpose": ""},
        # attention scores Q K^T of twelve heads, two heads per ciphertext
        {"name": "attention_qk", "kind": "product", "pairs": 6, "tiles": 2, "schedule": 2, "transpose": "right"},
        # one LoRA gradient (X A)^T dY over the three pairs of a 768-wide activation
        {"name": "lora_gradient", "kind": "product", "pairs": 3, "tiles": 2, "schedule": 2, "transpose": "left"},
        # score assembly of the Gaussian-kernel attention for one query / key pair, default schedule
        {"name": "gaussian_scores", "kind": "scores", "batch": 1, "schedule": 0},
        # the Q, K and V projections: 768 x 768 weights each on shared activations (a group of four tiles and one of two)
        {"name": "projection_qkv", "kind": "projection", "k_tiles": 6, "n_tiles": 18, "schedule": 2},
        # inputs of a few products entering, results leaving
        {"name": "encrypt_13", "kind": "encrypt", "count": 13, "level": 12},
        {"name": "decrypt_13", "kind": "decrypt", "count": 13, "level": 4},
        # the whole layer on resident operands, and from host matrices to host matrices
        {"name": "layer_resident", "kind": "layer", "end_to_end": False},
        {"name": "layer_end_to_end", "kind": "layer", "end_to_end": True},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["primitive", "primitive", "product", "product", "projection", "scores", "encrypt", "decrypt"])
    if kind == "primitive":
        op = rng.choice(["rotate", "mult", "rescale", "ntt", "intt"])
        return {"kind": kind, "op": op, "level": rng.randint(1, LEVELS), "batch": _log(rng, 1, 256), "step": rng.choice([1, 128, 4096]) if op == "rotate" else 0}
    if kind == "product":
        schedule = rng.choice([0, 1, 2, 2])
        return {"kind": kind, "pairs": _log(rng, 1, 20) if schedule == 2 else _log(rng, 1, 5), "tiles": rng.choice([1, 2]) if schedule == 0 else 2, "schedule": schedule,
                "transpose": rng.choice(["", "right", "left"])}
    if kind == "projection":
        return {"kind": kind, "k_tiles": _log(rng, 1, 24), "n_tiles": _log(rng, 1, 24), "schedule": rng.choice([0, 2, 2])}
    if kind == "scores":
        return {"kind": kind, "batch": rng.randint(1, 4), "schedule": rng.choice([0, 1, 2])}
    return {"kind": kind, "count": _log(rng, 1, 96), "level": rng.randint(TARGET, LEVELS) if kind == "encrypt" else rng.randint(1, 6)}


# ---- what a program holds for its whole life -----------------------------------------------------------------------
def _pkg():
    return importlib.import_module(PKG)


def _lib():
    if "lib" not in _held:
        _held["lib"] = _pkg().open_gpu(_pkg().make_params())
        _held["lib"].keygen()
    return _held["lib"]


def _hemmer(schedule):
    if schedule not in _held:
        _held[schedule] = _pkg().open_hemmer(_lib())
        _held[schedule].set_schedule(schedule)
    return _held[schedule]


class _Residues:
    """The device memory of a ciphertext handle, for torch; the handle lives as long as the tensor."""

    def __init__(self, ct):
        lib = ct.lib
        level, polys, batch, _ = lib.ct_meta(ct)
        address = lib._fn("ct_device_ptr")
        address.restype = importlib.import_module("ctypes").c_void_p
        self.ct = ct
        self.__cuda_array_interface__ = {"shape": (batch, polys, level + 1, lib.N), "typestr": "<i8", "data": (address(ct.ptr), False), "version": 3, "strides": None}


def _tensor(ct):
    return torch.as_tensor(_Residues(ct), device="cuda")


# ---- inputs --------------------------------------------------------------------------------------------------------
def _uniform(lib, level, batch, seed, scale_pow=1):
    """A batch of ciphertexts with uniform residues below each prime."""
    ct = lib.ct_create(level, 2, batch, scale_pow)
    view, gen = _tensor(ct), torch.Generator(device="cuda").manual_seed(seed)
    for limb in range(level + 1):
        view[:, :, limb].random_(0, int(lib.primes[limb]), generator=gen)
    torch.cuda.synchronize()   # the library's stream does not wait for torch's
    return ct


def _rng(seed):
    return np.random.default_rng([seed, 20240])


def _pairs(rng, count):
    return [(rng.uniform(-1, 1, (D, D)), rng.uniform(-1, 1, (D, D))) for _ in range(count)]


def _nonces(seed, count, base=0):
    return [(seed + 1) * 1_000_000 + base + k for k in range(count)]


def _k_groups(k_tiles):
    """K tiles in groups of four: (groups with two operand pairs, groups with one), as lists of group numbers."""
    groups = range((k_tiles + 3) // 4)
    full = [g for g in groups if 4 * g + 2 < k_tiles]
    return full, [g for g in groups if g not in full]


def prepare(case, seed):
    lib, kind = _lib(), case["kind"]
    if _held.get("case") != case:   # other work than before: its buffer sizes are of no use to what follows
        lib._chk(lib._fn("release_cached")(lib.ctx))
        _held["case"] = dict(case)
    s = {"case": case, "lib": lib}
    rng = _rng(seed)
    if kind == "primitive":
        s["a"] = _uniform(lib, case["level"], case["batch"], seed, 2 if case["op"] == "rescale" else 1)
        if case["op"] == "mult":
            s["b"] = _uniform(lib, case["level"], case["batch"], seed + 1)
        if case["op"] == "rotate":
            lib.gen_rot_keys([case["step"]])
    elif kind in ("product", "scores"):
        h = s["h"] = _hemmer(case["schedule"])
        count = case["pairs"] if kind == "product" else case["batch"]
        if case.get("tiles", 2) == 2:
            s["a"], s["b"] = (h.encrypt2_many(_pairs(rng, count), _nonces(seed, count, base)) for base in (0, 1000))
        else:
            one = [[h.encrypt(rng.uniform(-1, 1, (D, D)), nonce).ct for nonce in _nonces(seed, count, base)] for base in (0, 1000)]
            s["a"], s["b"] = (_pkg().CtxtTensor(lib.batch_concat(cts), D, D) for cts in one)
    elif kind == "projection":
        h = s["h"] = _hemmer(case["schedule"])
        k, n = case["k_tiles"], case["n_tiles"]
        zero = np.zeros((D, D))
        x = [rng.uniform(-1, 1, (D, D)) if t < k else zero for t in range(k + 3)]
        w = [[rng.normal(0.0, 0.02, (D, D)) if t < k else zero for t in range(k + 3)] for _ in range(n)]
        full, half = _k_groups(k)
        enc = lambda groups, off: h.encrypt2_many([(x[4 * g + off], x[4 * g + off + 1]) for g in groups], [_nonces(seed, 1, 4 * g + off)[0] for g in groups])
        pts = lambda groups: [[h.encode_diagonal_to_row4(*w[j][4 * g:4 * g + 4], level=TARGET + 1) for g in groups] for j in range(n)]
        s["full"] = (enc(full, 0), enc(full, 2), pts(full)) if full else None
        s["half"] = (enc(half, 0), None, pts(half)) if half else None
    elif kind == "encrypt":
        s["h"], s["nonces"] = _hemmer(2), _nonces(seed, case["count"])
        s["messages"] = np.stack([rng.uniform(-1, 1, lib.slots) for _ in range(case["count"])])
        s["pairs"] = [(m.reshape(D, 2 * D)[:, :D].copy(), m.reshape(D, 2 * D)[:, D:].copy()) for m in s["messages"]]
    elif kind == "decrypt":
        messages = np.stack([rng.uniform(-1, 1, lib.slots) for _ in range(case["count"])])
        ct = lib.encrypt_many(messages, case["level"], _nonces(seed, case["count"]))
        s["items"] = [(ct, k) for k in range(case["count"])]
    else:
        layer = importlib.import_module(PKG + ".layer")
        s["layer"] = layer.LayerWorkload(_hemmer(2), layer.synthetic(seed))
        s["layer"].prepare()   # encodes the weights and makes the operands resident
        if case["end_to_end"]:
            s["layer"].resident = None
    lib.sync()
    return s


# ---- one pass ------------------------------------------------------------------------------------------------------
def run(s):
    case, lib, kind = s["case"], s["lib"], s["case"]["kind"]
    if kind == "primitive":
        op = case["op"]
        if op == "rotate":
            return _tensor(lib.rotate(s["a"], case["step"]))
        if op == "mult":
            return _tensor(lib.mul(s["a"], s["b"]))
        if op == "rescale":
            return _tensor(lib.rescale(s["a"]))
        copy = lib.batch_slice(s["a"], 0, case["batch"])   # the transform works in place: on a copy, so that every pass sees the same input
        lib.ntt(copy, inverse=op == "intt")
        return _tensor(copy)
    if kind == "product":
        h, pair = s["h"], []
        for side, name in (("a", "left"), ("b", "right")):
            t = _pkg().CtxtTensor(s[side].ct, *s[side].shape)
            if case["transpose"] == name:
                # the fast schedule transposes at the lowest level that the product needs, as layer.py does
                h.transpose_inplace(t, TARGET + 3 if case["schedule"] == 2 else 0)
            pair.append(t)
        return _tensor(h.single_cc_matmul(*pair, TARGET).ct)
    if kind == "scores":
        return [_tensor(t.ct) for t in s["h"].gaussian_kernel_scores(s["a"], s["b"], TARGET)]
    if kind == "projection":
        h, outs = s["h"], None
        for first, second, weights in filter(None, (s["full"], s["half"])):
            packed = h.complex_packing(first, second) if second is not None else first
            groups = len(weights[0])
            parts = [t.ct for t in h.matmul_reuse_groups_tiles(h.matmul_pre(packed, TARGET), groups, 0, weights)]
            outs = parts if outs is None else [lib.add(a, b) for a, b in zip(outs, parts)]
        return [_tensor(ct) for ct in outs]
    if kind == "encrypt":
        if case["level"] == LEVELS:
            return _tensor(s["h"].encrypt2_many(s["pairs"], s["nonces"]).ct)
        return _tensor(lib.encrypt_many(s["messages"], case["level"], s["nonces"]))
    if kind == "decrypt":
        return lib.decrypt_many(s["items"])
    layer = s["layer"]
    if case["end_to_end"]:
        layer.step_e2e()
        tiles = {}
        for tag, value in layer.results:   # output tiles of one weight matrix side by side; every ct x ct product on its own
            tiles.setdefault(tag[1:3] if tag[0] == "p" else tag, []).append(value)
        return [np.concatenate(v, axis=1) if len(v) > 1 else v[0] for v in tiles.values()]
    out = layer.step_resident()
    return [_tensor(t.ct) for t in out["pcmm"].values()] + [_tensor(t.ct) for _, t in out["ccmm"].values()]


# ---- what a pass cannot do without ---------------------------------------------------------------------------------
def _switch(level):
    """(limbs of the switching key, modular products per ciphertext) of one key switch."""
    n, digits = level + 1, (level + 1) // ALPHA + 1
    ext = n + SPECIAL
    lifted = digits * ext - n
    transforms = n + lifted + 2 * SPECIAL + 2 * n
    return 2 * digits * ext, transforms * (N // 2) * 16 + 2 * digits * ext * N


def _product_work(pairs):
    """(limbs of operands and results, limbs of the distinct keys, modular products) of `pairs` tile products: two hoisted sets
    of shifted copies (127 each, one division by P q_l per copy) and the transforms before them (about 60 rotations)."""
    level = TARGET + 2
    limbs, ops = _switch(level)
    n, ext, digits = level + 1, level + 1 + SPECIAL, (level + 1) // ALPHA + 1
    copy = (2 * (SPECIAL + 1) + 2 * level) * (N // 2) * 16 + 3 * digits * ext * N
    keys = (3 * (D - 1) + 60) * limbs
    return pairs * 2 * (2 * (LEVELS + 1) + TARGET + 1), keys, pairs * (2 * (D - 1) * copy + 62 * ops)


def _projection_work(cts, groups, n_tiles):
    limbs, keys, ops = _product_work(1)
    level = TARGET + 1
    moved = cts * 2 * (LEVELS + 1) + n_tiles * (groups + 2) * (level + 1)
    return moved, keys // 2, groups * ops // 2 + groups * n_tiles * D * 2 * (level + 1) * N


def work(case):
    kind = case["kind"]
    if kind == "primitive":
        n, b, op = case["level"] + 1, case["batch"], case["op"]
        limbs, ops = _switch(case["level"])
        if op == "rotate":
            limbs, ops = limbs + b * 4 * n, b * ops
        elif op == "mult":
            limbs, ops = limbs + b * (6 * n - 2), b * (ops + 4 * n * N + 2 * n * (N // 2) * 16)
        elif op == "rescale":
            limbs, ops = b * (4 * n - 2), b * 2 * n * (N // 2) * 16
        else:
            limbs, ops = b * 4 * n, b * 2 * n * (N // 2) * 16
    elif kind == "product":
        limbs, keys, ops = _product_work(case["pairs"])
        limbs += keys if case["schedule"] else 0
    elif kind == "scores":
        limbs, _, ops = _product_work(case["batch"])
        limbs, ops = limbs + _switch(LEVELS)[0] * 20, 2 * ops
    elif kind == "projection":
        full, half = _k_groups(case["k_tiles"])
        limbs, keys, ops = _projection_work(2 * len(full) + len(half), len(full) + len(half), case["n_tiles"])
        limbs += keys if case["schedule"] else 0
    elif kind in ("encrypt", "decrypt"):
        # the host's values once, the ciphertext once; an embedding and its transforms
        n = case["level"] + 1 if kind == "encrypt" else 2
        limbs = case["count"] * (2 * n + 1)
        ops = case["count"] * ((N // 4) * 15 * 4 + (2 * n if kind == "encrypt" else n) * (N // 2) * 16)
    else:
        a, keys, ops = _product_work(42)
        limbs = a + keys
        for cts, groups, tiles in ((3, 2, 18), (3, 2, 6), (3, 2, 24), (12, 6, 6)):
            p, _, more = _projection_work(cts, groups, tiles)
            limbs, ops = limbs + p, ops + more
    return {"bytes": 8 * N * limbs, "flops": 2 * ops}


def tolerance(case):
    # decrypted values: a double-precision transform of 2^15 points; everything else is whole numbers
    if case["kind"] == "decrypt" or case.get("end_to_end"):
        return {"rel": 1e-13}
    return "exact"
