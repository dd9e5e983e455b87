"""The work a user of the engine has it do, as cases that can be timed: programmable bootstraps from one ciphertext to
the largest batches, on both parameter sets and with packed LUTs, the reference's own operator surface, whole Spike-LSTM
timesteps on both tori, a serving tick, and the two operators between bootstraps.

Inputs are made on the GPU from the seed alone; keys and models are those of one server (made once, as a server keeps
them), so another seed means other ciphertexts under the same keys.

All outputs but the operator surface's are torus words, whole numbers modulo q.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "blind-spiking-lstm_b200"))

from tfhe_b200 import client, ops  # noqa: E402
from tfhe_b200 import spike_model as SM  # noqa: E402
from tfhe_b200.engine import Keys  # noqa: E402
from tfhe_b200.params import CONFIG1, CONFIG2  # noqa: E402
from tfhe_b200.serving import DeviceStepModel  # noqa: E402

KEY_SEED = 2024
SETS = {"n630": (CONFIG1, 16, 32), "n742": (CONFIG2, 8, 8)}  # parameters, messages Z_t, output scale q / t_out


def listed():
    return [
        # one encrypted bit on its own: the latency of a single gate
        {"name": "pbs_n630_b1", "kind": "pbs", "set": "n630", "batch": 1, "n_lut": 1, "own_lut": False},
        # the plain bootstrap workload: 256 ciphertexts against one step LUT
        {"name": "pbs_n630_b256", "kind": "pbs", "set": "n630", "batch": 256, "n_lut": 1, "own_lut": False},
        # many-LUT bootstraps of an odd batch: four packed outputs per blind rotation
        {"name": "pbs_n630_lut4_b3001", "kind": "pbs", "set": "n630", "batch": 3001, "n_lut": 4, "own_lut": False},
        # the N = 2048 throughput sweep, each ciphertext with its own LUT: small, middle and large batch
        {"name": "pbs_n742_b64", "kind": "pbs", "set": "n742", "batch": 64, "n_lut": 1, "own_lut": True},
        {"name": "pbs_n742_b1024", "kind": "pbs", "set": "n742", "batch": 1024, "n_lut": 1, "own_lut": True},
        {"name": "pbs_n742_b16384", "kind": "pbs", "set": "n742", "batch": 16384, "n_lut": 1, "own_lut": True},
        # a caller of the reference's operators (float64 values, keys passed on every call)
        {"name": "cuboot_n630_b32", "kind": "cuboot", "batch": 32, "n_lut": 4},
        # a serving tick: two layers of 256 units, two requests in the first and one in the second
        {"name": "tick_h256_2_1", "kind": "tick", "first": 2, "second": 1},
        # one timestep of the one-layer model (hidden 128, embedding 64) for 16 sequences, on each torus
        {"name": "step32_s16", "kind": "step", "torus": 32, "seqs": 16},
        {"name": "step64_s16", "kind": "step", "torus": 64, "seqs": 16},
        # the operators between bootstraps on the 2^64 torus: LWEs into RLWEs by the trace, and by the packing key
        {"name": "trace64_r512", "kind": "trace", "rows": 512},
        {"name": "pack64_s16_t128", "kind": "pack", "seqs": 16, "lwes": 128},
    ]


def _spread(rng, lo, hi):
    """A whole number in [lo, hi], even over the logarithm, odd as often as not."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["pbs", "pbs", "pbs", "cuboot", "tick", "step", "trace", "pack"])
    if kind == "pbs":
        return {"kind": kind, "set": rng.choice(list(SETS)), "batch": _spread(rng, 1, 8192), "n_lut": rng.choice([1, 2, 4]),
                "own_lut": rng.random() < 0.5}
    if kind == "cuboot":
        return {"kind": kind, "batch": _spread(rng, 1, 512), "n_lut": rng.choice([1, 2, 4])}
    if kind == "tick":
        return {"kind": kind, "first": rng.randint(1, 6), "second": rng.randint(1, 6)}
    if kind == "step":
        return {"kind": kind, "torus": rng.choice([32, 64]), "seqs": _spread(rng, 1, 40)}
    if kind == "trace":
        return {"kind": kind, "rows": _spread(rng, 16, 4096)}
    return {"kind": kind, "seqs": _spread(rng, 1, 40), "lwes": _spread(rng, 16, 256)}


# ---------------------------------------------------------------- what a server keeps
@functools.lru_cache(maxsize=None)
def _client_keys(name):
    return client.keygen(SETS[name][0], KEY_SEED)


@functools.lru_cache(maxsize=None)
def _keys(name):
    k = _client_keys(name)
    return Keys.create(SETS[name][0], k.bsk, k.ksk_a, k.ksk_b)


@functools.lru_cache(maxsize=None)
def _model(torus, layers, hidden):
    cfg = SM.config_q64(layers=layers, hidden=hidden) if torus == 64 else SM.SpikeModelConfig(layers=layers, hidden=hidden)
    model = SM.build_model(cfg, seed=KEY_SEED)
    return model, SM.to_device(model)


@functools.lru_cache(maxsize=None)
def _server():
    model, dm = _model(32, 2, 256)
    step = DeviceStepModel(dm)
    step.warm_graphs(4)
    return model, step


@functools.lru_cache(maxsize=None)
def _reference_keys():
    """The n = 630 keys as the reference holds them: complex128 key spectra (2 out, 2 in, l, G M, N/2), the monomials' spectra,
    float64 key-switching key."""
    p, k = CONFIG1, _client_keys("n630")
    twist = torch.exp(-1j * math.pi * torch.arange(p.N, device="cuda", dtype=torch.float64) / p.N)
    bsk = torch.from_numpy(client._centred(k.bsk)).cuda().to(torch.float64)  # (2, 2, G M, l, N)
    four = torch.empty((2, 2, p.l_bs, p.G * p.M, p.N // 2), dtype=torch.complex128, device="cuda")
    for side in range(2):
        for out in range(2):
            four[out, side] = torch.fft.fft(bsk[side, out] * twist)[..., : p.N // 2].permute(1, 0, 2)
    angle = (torch.arange(2 * p.N, device="cuda")[:, None] * (2 * torch.arange(p.N // 2, device="cuda") + 1)) % (2 * p.N)
    rot = torch.exp(-1j * math.pi * angle.to(torch.float64) / p.N)
    ksk = (torch.from_numpy(client._centred(k.ksk_a)).cuda().to(torch.float64),
           torch.from_numpy(client._centred(k.ksk_b)).cuda().to(torch.float64).unsqueeze(-1))
    return four, rot, ksk


# ---------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _lwes32(p, sk, batch, t, seed):
    """LWEs under the GLWE key of uniform messages in Z_t with a padding bit, as int32 words on the GPU."""
    g = _generator(seed)
    a = torch.randint(-(2 ** 31), 2 ** 31, (batch, p.big), device="cuda", generator=g, dtype=torch.int64)
    s = torch.from_numpy(np.asarray(sk, dtype=np.float64)).cuda()
    m = torch.randint(0, t, (batch,), device="cuda", generator=g)
    e = torch.round(torch.randn((batch,), device="cuda", generator=g, dtype=torch.float64) * p.sigma_glwe).to(torch.int64)
    b = torch.empty((batch,), dtype=torch.int64, device="cuda")
    for o in range(0, batch, 2048):
        b[o:o + 2048] = (a[o:o + 2048].to(torch.float64) @ s).to(torch.int64)
    b += m * (2 ** 32 // (2 * t)) + e
    return a.to(torch.int32), b.to(torch.int32)


def _lwes64(sk, shape, seed):
    """LWEs of spikes (0 or 1 at scale 2^54) under the GLWE key, as int64 words on the GPU."""
    g = _generator(seed)
    s = torch.from_numpy(np.asarray(sk, dtype=np.int64)).cuda()
    hi = torch.randint(-(2 ** 31), 2 ** 31, shape + (s.numel(),), device="cuda", generator=g, dtype=torch.int64)
    a = hi * 2 ** 32 + torch.randint(0, 2 ** 32, hi.shape, device="cuda", generator=g, dtype=torch.int64)
    e = torch.randint(-(2 ** 18), 2 ** 18, shape, device="cuda", generator=g, dtype=torch.int64)
    return a, (a * s).sum(-1) + torch.randint(0, 2, shape, device="cuda", generator=g) * 2 ** 54 + e


def _luts32(p, t, t_out, n_lut, count, seed):
    """LUT polynomials (count, 2, N): random tables Z_t -> Z_t_out/2, n_lut of them packed per polynomial."""
    rng = np.random.default_rng(seed)
    pool = [client.packed_table_lut(p.N, rng.integers(0, t_out // 2, size=(n_lut, t)), t_out) for _ in range(min(8, count))]
    pool = torch.from_numpy(np.stack(pool).view(np.int32)).cuda()
    lut = torch.zeros((count, 2, p.N), dtype=torch.int32, device="cuda")
    lut[:, 1] = pool[torch.from_numpy(rng.integers(0, len(pool), size=count)).cuda()]
    return lut


def _layer_inputs(model, layer, seqs, seed):
    """The encrypted inputs of one timestep of a layer, and its states after earlier ones: hidden spikes and cell values."""
    cfg, rng = model.cfg, np.random.default_rng(seed)
    L = model.layers[layer]
    cl = SM.client64 if cfg.torus_bits == 64 else client

    def encrypt(values, at):
        poly = np.zeros((seqs, cfg.pbs.N), dtype=np.int64)
        poly[:, at:at + values.shape[1]] = values * cfg.beta_x
        a, b = cl.encrypt_rlwe(poly, model.keys.sk_glwe, cfg.sigma_rlwe, rng)
        return SM.encrypted_words(model, np.stack([a, b], axis=1)).cuda()

    if layer == 0:
        tokens = SM.sample_tokens(rng, seqs, 1, cfg.vocab, cfg.zipf)
        x = SM.encrypted_words(model, SM.encrypt_tokens(model, tokens, rng)).cuda()[0].contiguous()
    else:
        x = encrypt(rng.integers(0, 2, size=(seqs, cfg.hidden)), 0)
    H = encrypt(rng.integers(0, 2, size=(seqs, cfg.hidden)), L.in_dim)
    C = encrypt(rng.integers(0, 3, size=(seqs, cfg.hidden)), 0)
    return x, H, C


def prepare(case, seed):
    kind = case["kind"]
    if kind == "pbs":
        p, t, t_out = SETS[case["set"]]
        a, b = _lwes32(p, _client_keys(case["set"]).sk_glwe, case["batch"], t, seed)
        lut = _luts32(p, t, t_out, case["n_lut"], case["batch"] if case["own_lut"] else 1, seed)
        return {"kind": kind, "keys": _keys(case["set"]), "a": a, "b": b, "lut": lut, "n_lut": case["n_lut"]}
    if kind == "cuboot":
        p, t, t_out = SETS["n630"]
        four, rot, ksk = _reference_keys()
        a, b = _lwes32(p, _client_keys("n630").sk_glwe, case["batch"], t, seed)
        lut = _luts32(p, t, t_out, case["n_lut"], case["batch"], seed).to(torch.float64)
        boot = ops.HeavysideBoostrapper(
            four, ksk, None, None, {"q": 2 ** 32},
            {"q": 2 ** 32, "beta_bs": 2 ** p.log2_beta_bs, "l_bs": p.l_bs, "degree": p.N},
            {"q": 2 ** 32, "beta_ks": 2 ** p.log2_beta_ks, "l_ks": p.l_ks}, None, p.collapse, rot, case["n_lut"])
        return {"kind": kind, "boot": boot, "h": (a.to(torch.float64), b.to(torch.float64).unsqueeze(-1)),
                "lut": (lut[:, 0].contiguous(), lut[:, 1].contiguous())}
    if kind == "tick":
        model, step = _server()
        parts = [_layer_inputs(model, l, n, seed + 7919 * l) for l, n in enumerate((case["first"], case["second"]))]
        return {"kind": kind, "step": step, "xs": [x for x, _, _ in parts],
                "states": [torch.stack([H, C], dim=1) for _, H, C in parts]}
    if kind == "step":
        model, dm = _model(case["torus"], 1, 128)
        x, H, C = _layer_inputs(model, 0, case["seqs"], seed)
        return {"kind": kind, "layer": dm.layers[0], "x": x, "H": H, "C": C}
    model, dm = _model(64, 1, 128)
    shape = (case["rows"],) if kind == "trace" else (case["seqs"], case["lwes"])
    a, b = _lwes64(model.keys.sk_glwe, shape, seed)
    return {"kind": kind, "keys": dm.keys, "a": a, "b": b}


# ---------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "pbs":
        return state["keys"].pbs(state["a"], state["b"], state["lut"], state["n_lut"])
    if kind == "cuboot":
        return state["boot"].cuboot(state["h"], state["lut"])
    if kind == "tick":
        return state["step"].step_layers(state["xs"], state["states"])
    if kind == "step":
        return state["layer"].step(state["x"], state["H"], state["C"])
    if kind == "trace":
        return state["keys"].galois.pack_lwe_to_rlwe(state["a"], state["b"])
    return state["keys"].pack(state["a"], state["b"])


# ---------------------------------------------------------------- what a pass cannot do without
def _transform(N):
    return 5 * (N // 2) * math.log2(N // 2)


def _rotations(p, count, n_lut, word):
    """Blind rotations with their key switch: FP64 operations of the transforms and of the key products, the two keys
    read once (the bootstrapping key as double spectra), each ciphertext and LUT in, its extractions out."""
    h, P = p.N // 2, 2 * p.l_bs
    flops = p.G * ((P + 2) * _transform(p.N) + 8 * h * (2 * P * p.M + P))
    switch = 2 * p.big * p.l_ks * (p.n + 1)
    keys = p.G * 2 * P * p.M * h * 16 + p.big * p.l_ks * (p.n + 1) * word
    return count * (flops + switch), keys + count * word * (p.big + 1 + 2 * p.N + n_lut * (p.N + 1))


def _packing(cfg, rows, seqs, word):
    N, l = cfg.pbs.N, cfg.pk_l
    return 2 * rows * N * l * 2 * N, N * l * 2 * N * word + rows * (N + 1) * word + seqs * 2 * N * word


def _trace(cfg, rows, word):
    """The Galois key has 16-bit limbs on the 2^64 torus, each product its own inverse transform."""
    N, l, limbs = cfg.pbs.N, cfg.gal_l, 4 if word == 8 else 1
    steps = int(math.log2(N))
    flops = rows * steps * ((l + 2 * limbs) * _transform(N) + 8 * (N // 2) * l * 2 * limbs)
    return flops, steps * l * 2 * N * word + rows * (N + 1 + 2 * N) * word


def _layer(cfg, seqs, in_dim):
    """One timestep of `seqs` sequences: three linears, two LUT preparations, 3 hidden / n_lut rotations, two packings."""
    word, N, per = cfg.torus_bits // 8, cfg.pbs.N, cfg.hidden // cfg.n_lut
    parts = [_rotations(cfg.pbs, 3 * per * seqs, cfg.n_lut, word), _packing(cfg, 2 * cfg.hidden * seqs, 2 * seqs, word),
             _trace(cfg, 2 * cfg.hidden * seqs, word)]
    flops = 3 * per * seqs * 2 * (in_dim + cfg.hidden) * N + 2 * cfg.hidden * seqs * 3 * _transform(N)
    return sum(f for f, _ in parts) + flops, sum(b for _, b in parts)


def work(case):
    kind = case["kind"]
    if kind == "pbs":
        flops, moved = _rotations(SETS[case["set"]][0], case["batch"], case["n_lut"], 4)
    elif kind == "cuboot":
        flops, moved = _rotations(CONFIG1, case["batch"], case["n_lut"], 8)
    elif kind == "tick":
        cfg = SM.SpikeModelConfig(layers=2, hidden=256)
        parts = [_layer(cfg, case["first"], cfg.emb_dim), _layer(cfg, case["second"], cfg.hidden)]
        flops, moved = sum(f for f, _ in parts), parts[0][1]
    elif kind == "step":
        cfg = SM.config_q64() if case["torus"] == 64 else SM.SpikeModelConfig()
        flops, moved = _layer(cfg, case["seqs"], cfg.emb_dim)
    elif kind == "trace":
        flops, moved = _trace(SM.config_q64(), case["rows"], 8)
    else:
        flops, moved = _packing(SM.config_q64(), case["seqs"] * case["lwes"], case["seqs"], 8)
    return {"bytes": moved, "flops": flops}


# ---------------------------------------------------------------- in 64 bits
def _wrap(x):
    """int64 -> centred modulo 2^32."""
    return ((x + 2 ** 31) & (2 ** 32 - 1)) - 2 ** 31


def _digits(x, log2_beta, levels):
    """The gadget digits of centred values (float64), first level first: x = value / q, d = round(beta x)."""
    x, out = x.to(torch.float64) / 2.0 ** 32, []
    for _ in range(levels):
        y = x * 2.0 ** log2_beta
        out.append(torch.round(y))
        x = y - out[-1]
    return out


def _exact_bootstrap(p, keys, a, b, lut, n_lut):
    """Key switch, collapsed blind rotation, rotation by -b~ and extraction of LWEs a (B, n_big), b (B) against LUTs
    (B, 2, N), all int64: every product here is a whole number that float64 holds, so the words are exact."""
    B, N, n, M = a.shape[0], p.N, p.n, p.M
    ka = torch.from_numpy(client._centred(keys.ksk_a)).cuda().to(torch.float64)
    kb = torch.from_numpy(client._centred(keys.ksk_b)).cuda().to(torch.float64)
    sa, sb = torch.zeros((B, n), dtype=torch.float64, device="cuda"), b.to(torch.float64)
    for j, d in enumerate(_digits(a, p.log2_beta_ks, p.l_ks)):
        sa, sb = sa + d @ ka[j], sb + d @ kb[j]
    sa, sb = _wrap(sa.to(torch.int64)), _wrap(sb.to(torch.int64))
    pattern = torch.tensor([[(m >> (p.collapse - 1 - c)) & 1 for c in range(p.collapse)] for m in range(M)], device="cuda")
    sums = (sa.view(B, p.G, 1, p.collapse) * pattern).sum(-1).to(torch.float64)
    turn = (torch.round(2 * N * sums / (2.0 ** 32 * n_lut)) * n_lut).to(torch.int64) % (2 * N)
    at = torch.arange(N, device="cuda")
    twist = torch.exp(-1j * math.pi * at.to(torch.float64) / N)
    bsk = torch.from_numpy(client._centred(keys.bsk)).cuda().view(2, 2, p.G, M, p.l_bs, N)
    acc = lut.clone()
    point = 2 * torch.arange(N, device="cuda") + 1
    for g in range(p.G):
        dec = torch.stack(_digits(acc, p.log2_beta_bs, p.l_bs), dim=1)  # (B, l, 2, N)
        spectrum = torch.fft.fft(dec * twist)
        key = torch.fft.fft(bsk[:, :, g].to(torch.float64) * twist)  # (in, out, M, l, N)
        total = torch.zeros((B, 2, N), dtype=torch.complex128, device="cuda")
        for m in range(M):
            angle = (turn[:, g, m, None] * point) % (2 * N)
            total += torch.exp(-1j * math.pi * angle.to(torch.float64) / N)[:, None] * torch.einsum("bljn,joln->bon", spectrum, key[:, :, m])
        acc = _wrap(torch.round((torch.fft.ifft(total) * twist.conj()).real).to(torch.int64))
    bt = (torch.round(2 * N * sb.to(torch.float64) / (2.0 ** 32 * n_lut)) * n_lut).to(torch.int64)

    def coefficient(poly, e):
        e = e % (2 * N)
        v = torch.gather(poly, 1, e % N)
        return torch.where(e < N, v, _wrap(-v))

    j = torch.arange(n_lut, device="cuda")
    out_a = torch.stack([coefficient(acc[:, 0], i - at[None] + bt[:, None]) for i in range(n_lut)], dim=1)
    return out_a, coefficient(acc[:, 1], j[None] + bt[:, None])


def exact(case, seed):
    """The bootstraps at gadget base 2^7, whose products float64 holds exactly.  At base 2^15, and on the 2^64 torus, the
    float64 transforms round, so a chain's words are a sample of its noise and 64 bits give no other value for them; the
    remaining outputs are whole numbers."""
    if case["kind"] not in ("pbs", "cuboot") or case.get("set", "n630") != "n630" or case["batch"] > 256:
        return None
    s = prepare(case, seed)
    p, keys = CONFIG1, _client_keys("n630")
    if case["kind"] == "pbs":
        lut = s["lut"].to(torch.int64).expand(case["batch"], 2, p.N)
        a, b = _exact_bootstrap(p, keys, s["a"].to(torch.int64), s["b"].to(torch.int64), lut, s["n_lut"])
        return a.to(torch.int32), b.to(torch.int32)
    lut = torch.stack(s["lut"], dim=1).to(torch.int64)
    a, b = _exact_bootstrap(p, keys, s["h"][0].to(torch.int64), s["h"][1][:, 0].to(torch.int64), lut, case["n_lut"])
    return a.to(torch.float64), b.to(torch.float64).unsqueeze(-1)
