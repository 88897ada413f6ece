"""Workloads of the batched Classic McEliece KEM engine, as its users run them.

Each case goes through the package's public calls: batched encapsulation and
decapsulation against resident keys (device and host buffers), the one-request
libmceliece-shaped calls, a grouped plan over several keys and parameter sets,
constant-time decapsulation, and key generation. Sizes follow the repository's
benchmark (256 .. 65536 requests per batch, the Zipf mix over eight keys, key
batches) and its tests (single calls, ragged batches). One decapsulation input
in ten carries a flipped bit, as in the benchmark, so both outcomes run.
Every output is bytes or return codes: there are no computed real numbers, so
there is no 64-bit reference to define.
"""
import hashlib
import math

import numpy as np
import torch

import tensormceliece_gb300 as gmc

FLIP = 0.10  # share of decapsulation inputs with one flipped bit
# the grouped mix: eight keys over the five sets (348864, 460896, 6688128, 6960119, 8192128)
MIX = ("8192128", "348864", "6960119", "460896", "6688128", "348864", "8192128", "460896")
SETS = gmc.SETS


def listed():
    return [
        # a handshake server that decapsulates one ciphertext per call through the libmceliece convention
        {"name": "one_dec_8192128", "kind": "one_dec", "set": "8192128", "n": 1},
        # a client encapsulating once against a resident key, host buffers
        {"name": "host_enc_348864_n1", "kind": "host_enc", "set": "348864", "n": 1},
        # the benchmark's smallest configuration: 256 encapsulations and 256 decapsulations per step
        {"name": "kem_348864_n256", "kind": "kem", "set": "348864", "n": 256},
        # a batch of ordinary size that fills no tile evenly
        {"name": "enc_6960119_n3001", "kind": "enc", "set": "6960119", "n": 3001},
        # ordinary decapsulation batch, odd size
        {"name": "dec_460896_n9973", "kind": "dec", "set": "460896", "n": 9973},
        # plaintext confirmation through host buffers (a service that keeps its requests in host memory)
        {"name": "host_dec_6688128pc_n20000", "kind": "host_dec", "set": "6688128pc", "n": 20000},
        # the headline step's two halves
        {"name": "enc_8192128_n65536", "kind": "enc", "set": "8192128", "n": 65536},
        {"name": "dec_8192128_n65536", "kind": "dec", "set": "8192128", "n": 65536},
        # constant-time decapsulation, for a GPU shared with other tenants
        {"name": "dec_ct_8192128_n8192", "kind": "dec_ct", "set": "8192128", "n": 8192},
        # many tenants' keys in one launch: 65536 requests over eight keys
        {"name": "plan_mix_n65536", "kind": "plan", "set": "mix", "n": 65536},
        # one key pair on demand
        {"name": "keypair_8192128_n1", "kind": "keypair", "set": "8192128", "n": 1},
        # provisioning a fleet of keys in one call (semi-systematic form)
        {"name": "keypair_460896f_n200", "kind": "keypair", "set": "460896f", "n": 200},
    ]


def draw(rng):
    kind = rng.choice(("enc", "dec", "kem", "enc", "dec", "host_enc", "host_dec", "dec_ct", "plan", "keypair", "one_dec"))
    name = rng.choice(SETS)
    if kind == "one_dec":
        return {"kind": kind, "set": name + rng.choice(("", "pc")), "n": 1}
    if kind == "keypair":
        return {"kind": kind, "set": name + rng.choice(("", "f")), "n": _log_uniform(rng, 1, 48)}
    if kind == "plan":
        return {"kind": kind, "set": "mix", "n": _log_uniform(rng, 1024, 65536)}
    hi = {"dec_ct": 8192, "host_enc": 20000, "host_dec": 20000, "kem": 32768}.get(kind, 65536)
    return {"kind": kind, "set": name + rng.choice(("", "", "pc")), "n": _log_uniform(rng, 1, hi)}


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _bytes(seed, tag, n):
    return np.frombuffer(hashlib.shake_256(b"%d:%s" % (int(seed), tag.encode())).digest(n), np.uint8)


def _device_seeds(seed, tag, n):
    return torch.from_numpy(_bytes(seed, tag, 32 * n).copy()).cuda()


def _ciphertexts(pub, seed, tag, n):
    """n valid ciphertexts on the device, a tenth of them with one uniformly chosen bit flipped."""
    cb = pub.sizes["ct_bytes"]
    s = _device_seeds(seed, tag, n)
    c = torch.empty((n, cb), dtype=torch.uint8, device="cuda")
    k = torch.empty((n, 32), dtype=torch.uint8, device="cuda")
    pub.enc_batch_dev(c.data_ptr(), k.data_ptr(), s.data_ptr(), n, 0, torch.cuda.current_stream().cuda_stream)
    g = np.random.default_rng([int(seed), n])
    rows = np.flatnonzero(g.random(n) < FLIP)
    bits = g.integers(0, pub.sizes["mt"], rows.size)
    rows, bits = torch.from_numpy(rows).cuda(), torch.from_numpy(bits).cuda()
    c[rows, bits >> 3] ^= (1 << (bits & 7)).to(torch.uint8)
    torch.cuda.synchronize()
    return c


def _keys(name, seed, tag="key"):
    return gmc.keypair(name, bytes(_bytes(seed, tag, 32)))


def _shares(total, parts, s=1.2):
    """Request counts of `parts` keys with Zipf(1.2) weights, summing to total."""
    w = np.arange(1, parts + 1) ** -s
    c = np.floor(total * w / w.sum()).astype(int)
    c[0] += total - c.sum()
    return [int(x) for x in c]


def prepare(case, seed):
    kind, name, n = case["kind"], case["set"], case["n"]
    st = {"kind": kind, "n": n, "set": name}
    if kind == "keypair":
        st["seeds"] = _bytes(seed, "keypair", 32 * n).reshape(n, 32).copy()
        return st
    if kind == "plan":
        st["keys"], st["bufs"], groups = [], [], []
        for i, (s, count) in enumerate(zip(MIX, _shares(n, len(MIX)))):
            pk, sk = _keys(s, seed, "key%d" % i)
            pub, sec = gmc.PublicKey(s, pk), gmc.SecretKey(s, sk)
            ne, nd = count // 2, count - count // 2
            cb = pub.sizes["ct_bytes"]
            b = {"seeds": _device_seeds(seed, "seeds%d" % i, ne), "cin": _ciphertexts(pub, seed, "in%d" % i, nd),
                 "c": torch.empty((ne, cb), dtype=torch.uint8, device="cuda"),
                 "k": torch.empty((ne, 32), dtype=torch.uint8, device="cuda"),
                 "kd": torch.empty((nd, 32), dtype=torch.uint8, device="cuda"),
                 "rc": torch.empty(nd, dtype=torch.int32, device="cuda")}
            groups.append((pub, ne, b["seeds"].data_ptr(), b["c"].data_ptr(), b["k"].data_ptr(), 0))
            groups.append((sec, nd, b["cin"].data_ptr(), 0, b["kd"].data_ptr(), b["rc"].data_ptr()))
            st["keys"].append((pub, sec))
            st["bufs"].append(b)
        st["plan"] = gmc.Plan(groups)
        return st
    pk, sk = _keys(name, seed)
    if kind in ("enc", "kem", "host_enc"):
        st["pub"] = gmc.PublicKey(name, pk)
    if kind != "enc" and kind != "host_enc":
        st["sec"] = None if kind == "one_dec" else gmc.SecretKey(name, sk)
        cts = _ciphertexts(gmc.PublicKey(name, pk), seed, "in", n)
        if kind in ("one_dec", "host_dec"):
            st["cts"] = cts.cpu().numpy()
            st["sk"] = sk
        else:
            st["cts"] = cts
            st["kd"] = torch.empty((n, 32), dtype=torch.uint8, device="cuda")
            st["rc"] = torch.empty(n, dtype=torch.int32, device="cuda")
    if kind == "host_enc":
        st["seeds"] = _bytes(seed, "seeds", 32 * n).copy()
    elif kind in ("enc", "kem"):
        st["seeds"] = _device_seeds(seed, "seeds", n)
        st["c"] = torch.empty((n, st["pub"].sizes["ct_bytes"]), dtype=torch.uint8, device="cuda")
        st["k"] = torch.empty((n, 32), dtype=torch.uint8, device="cuda")
    return st


def _enc(st, stream):
    st["pub"].enc_batch_dev(st["c"].data_ptr(), st["k"].data_ptr(), st["seeds"].data_ptr(), st["n"], 0, stream)


def _dec(st, stream):
    st["sec"].dec_batch_dev(st["kd"].data_ptr(), st["cts"].data_ptr(), st["n"], st["rc"].data_ptr(), stream)


def run(st):
    kind = st["kind"]
    if kind == "one_dec":
        rc, k = gmc.kem_dec(st["set"], st["cts"], st["sk"])
        return [int(rc), np.frombuffer(k, np.uint8)]
    if kind == "host_enc":
        return list(st["pub"].enc_batch(st["seeds"]))
    if kind == "host_dec":
        return list(st["sec"].dec_batch(st["cts"]))
    if kind == "keypair":
        return list(gmc.keypair_batch(st["set"], st["seeds"]))
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "plan":
        st["plan"].launch(stream)
        return [b[x] for b in st["bufs"] for x in ("c", "k", "kd", "rc")]
    if kind == "enc":
        _enc(st, stream)
        return [st["c"], st["k"]]
    if kind == "dec":
        _dec(st, stream)
        return [st["kd"], st["rc"]]
    if kind == "dec_ct":
        gmc.set_dec_constant_time(True)
        try:
            _dec(st, stream)
        finally:
            gmc.set_dec_constant_time(False)
        return [st["kd"], st["rc"]]
    _enc(st, stream)
    _dec(st, stream)
    return [st["c"], st["k"], st["kd"], st["rc"]]


KECCAK_OPS = 24 * 180  # 32-bit logic and shift operations of one Keccak-f[1600] permutation


def _enc_work(z, n):
    """Seeds and the public key in, ciphertexts and keys out; the expected draws of the seed chain and the key hash."""
    pre = 1 + z["n"] // 8 + z["ct_bytes"]
    full = z["n"] == 1 << z["m"]
    blocks = -(-(2 * z["t"] if full else 4 * z["t"]) // 136)
    distinct = math.exp(sum(math.log1p(-i / z["n"]) for i in range(z["t"])))
    hashes = blocks / distinct + pre // 136 + 1
    return {"bytes": n * (64 + z["ct_bytes"]) + z["pk_bytes"],
            "flops": n * (hashes * KECCAK_OPS + z["t"] * z["mt"] / 32)}


def _dec_work(z, n):
    """Ciphertexts and the secret key in, keys out; the 2t syndromes, 2t^2 field products of the key equation
    solver and the additive FFT's d 2^(m-1), 32 products at a time as m^2 logic operations, and the key hash."""
    pre = 1 + z["n"] // 8 + z["ct_bytes"]
    d = 6 if z["t"] <= 64 else 7
    products = 2 * z["t"] ** 2 + d * (1 << (z["m"] - 1))
    return {"bytes": n * (32 + z["ct_bytes"]) + z["sk_bytes"],
            "flops": n * ((pre // 136 + 1) * KECCAK_OPS + products * z["m"] ** 2 / 32 + 2 * z["mt"] * z["mt"] / 32)}


def _keypair_work(z, n):
    """One successful attempt per key: the seed expansion and the elimination of the mt x n matrix, 32 bits a word."""
    out = n * (z["pk_bytes"] + z["sk_bytes"])
    expand = (z["n"] // 8 + (4 << z["m"]) + 2 * z["t"] + 32) // 136 + 1
    return {"bytes": out + 32 * n, "flops": n * (expand * KECCAK_OPS + z["mt"] ** 2 * z["n"] / 64)}


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "plan":
        parts = []
        for s, count in zip(MIX, _shares(n, len(MIX))):
            z = gmc.set_sizes(gmc.set_id(s))
            parts += [_enc_work(z, count // 2), _dec_work(z, count - count // 2)]
    else:
        z = gmc.set_sizes(gmc.set_id(case["set"]))
        parts = []
        if kind in ("enc", "kem", "host_enc"):
            parts.append(_enc_work(z, n))
        if kind in ("dec", "kem", "host_dec", "dec_ct", "one_dec"):
            parts.append(_dec_work(z, n))
        if kind == "keypair":
            parts.append(_keypair_work(z, n))
    return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}


def exact(case, seed):
    """Outputs are bytes and return codes: nothing here has a value in real arithmetic."""
    return None
