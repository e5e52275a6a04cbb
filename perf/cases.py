"""Performance cases: the work users of this framework have it do.

Each case goes through the public entry points (the Python mirror of the C
ABI, or the C ABI itself where a caller owns its output buffers): proofs one
at a time from the smallest to the largest, stacked layouts, lock-step
batches, a served mix, batched verification, and the pieces a host prover
calls on its own (encoding, Merkle commitment and openings, claim and
sumcheck passes).  Inputs are uniform random KoalaBear elements, as the
reference harness draws its polynomials.  All outputs are field elements,
digests and proof bytes: whole numbers.
"""
import random
import weakref

import numpy as np
import torch

import whir_gb300 as W

P = W.P
JOHNSON = W.SOUNDNESS["JohnsonBound"]
UNIQUE = W.SOUNDNESS["UniqueDecoding"]
CAPACITY = W.SOUNDNESS["CapacityBound"]


# ---------------------------------------------------------------- the cases
def _proof(name, k, rate, claims, folding=4, soundness=JOHNSON, security=100, host=False,
           initial_reduction=1):
    return dict(name=name, kind="prove", k=k, folding=folding, rate=rate,
                initial_reduction=initial_reduction, soundness=soundness, security=security,
                claims=claims, host=host)


def listed():
    return [
        # the smallest proof of the smoke configuration: latency of a call
        _proof("prove_k12", 12, 1, 1),
        # one proof of the batched configuration's small shape
        _proof("prove_k16", 16, 2, 2),
        # the plain single-instance configuration, polynomial in pinned host memory
        _proof("prove_k20_host", 20, 1, 1, host=True),
        # the headline configuration: 2^24 evaluations, rate 1/4, 4 claims
        _proof("prove_k24", 24, 2, 4),
        # a zkVM-like layout: polynomials of mixed sizes stacked into one
        # commitment, unique decoding, folding 3 (rows of 8 and 32 words)
        dict(name="prove_stacked", kind="stack", sizes="17,16,16,14,13,9,9", folding=3, rate=2,
             soundness=UNIQUE, security=100),
        # lock-step proofs of equal shape (the batched configuration's small jobs)
        dict(name="batch_64xk16", kind="batch", k=16, folding=4, rate=2, claims=2, n=64,
             commit_only=False),
        # commitments alone, many at once (the batched-commitment configuration)
        dict(name="commit_16xk18", kind="batch", k=18, folding=4, rate=1, claims=0, n=16,
             commit_only=True),
        # a worker pool proving a mix of sizes, rates and claim counts at once
        dict(name="serve_mix", kind="serve", jobs=32, k_lo=14, k_hi=20, mix=1),
        # a batch of proofs of one shape checked together
        dict(name="verify_64xk16", kind="verify", k=16, folding=4, rate=2, claims=2, n=64),
        # the Merkle benchmark's base shape: 2^21 rows of 32 elements, with openings
        dict(name="merkle_2e21x32", kind="merkle", log_h=21, row_len=32, openings=100),
        # encoding on its own, a ragged input height and a width off the proofs' shapes
        dict(name="dft_ragged", kind="dft", log_h=19, h_in=200003, width=20),
        # the passes of one opening round as a host prover calls them one by one
        dict(name="pieces_k20", kind="pieces", k=20, kept=4, eqs=2, pows=60),
    ]


def draw(rng):
    kind = rng.choice(("prove", "prove", "stack", "batch", "serve", "verify", "merkle", "dft",
                       "pieces"))
    if kind == "prove":
        folding = rng.choice((4, 4, 4, 5, 6, 3, 2))
        rate = rng.choice((1, 2, 2, 3))
        top = {2: 18, 3: 20}.get(folding, 24 if rate <= 2 else 22)
        c = _proof("", rng.randint(10, top), rate, rng.randint(0, 4), folding,
                   rng.choice((JOHNSON, JOHNSON, CAPACITY, UNIQUE)), rng.choice((100, 100, 80)),
                   rng.random() < 0.3, rng.randint(1, 2))
        del c["name"]
        return c
    if kind == "stack":
        folding = rng.choice((3, 4))
        k = rng.randint(12, 20)
        sizes, room = [], 1 << k
        while len(sizes) < 2 or (len(sizes) < 12 and room > (1 << k) // 3):
            kp = rng.randint(max(folding, k - 9), k - 1)
            if (1 << kp) <= room:
                sizes.append(kp)
                room -= 1 << kp
        if room >= 1 << (k - 1):  # the layout has to reach past 2^(k-1) words
            sizes[0] = k - 1
            sizes.append(folding)
        return dict(kind="stack", sizes=",".join(map(str, sizes)), folding=folding,
                    rate=rng.randint(1, 2), soundness=rng.choice((JOHNSON, UNIQUE)),
                    security=100)
    if kind == "batch":
        k = rng.randint(12, 20)
        most = max(2, min(256, 1 << (23 - k)))
        n = max(2, int(round(2 ** rng.uniform(1, np.log2(most)))))
        commit = rng.random() < 0.4
        return dict(kind="batch", k=k, folding=rng.choice((4, 4, 5)), rate=rng.randint(1, 2),
                    claims=0 if commit else rng.randint(1, 4), n=n, commit_only=commit)
    if kind == "serve":
        lo = rng.randint(12, 16)
        return dict(kind="serve", jobs=rng.randint(8, 40), k_lo=lo, k_hi=lo + rng.randint(1, 4),
                    mix=rng.randint(2, 1 << 20))
    if kind == "verify":
        return dict(kind="verify", k=rng.randint(12, 18), folding=rng.choice((3, 4, 5)),
                    rate=rng.randint(1, 2), claims=rng.randint(1, 3),
                    n=int(round(2 ** rng.uniform(3, 7))))
    if kind == "merkle":
        row_len = rng.choice((16, 32, 64, 128, 8, 4, rng.randint(1, 200)))
        log_h = rng.randint(8, min(21, 22 - max(0, -(-row_len // 16) - 1).bit_length()))
        return dict(kind="merkle", log_h=log_h, row_len=row_len, openings=rng.randint(1, 300))
    if kind == "dft":
        width = rng.choice((8, 16, 32, 64, 128, 4, 4 * rng.randint(1, 20), rng.randint(1, 40)))
        log_h = rng.randint(6, min(22, 27 - (width - 1).bit_length()))
        h_in = int(2 ** rng.uniform(log_h - 3, log_h))
        if rng.random() < 0.5:
            h_in = 1 << max(0, h_in.bit_length() - 1)
        return dict(kind="dft", log_h=log_h, h_in=max(1, h_in), width=width)
    return dict(kind="pieces", k=rng.randint(10, 24), kept=rng.randint(3, 6),
                eqs=rng.randint(1, 6), pows=rng.randint(1, 150))


# ---------------------------------------------------------------- what a program keeps
_keep = {}
_shared = weakref.WeakValueDictionary()  # provers and pools, while a state uses them


def _ctx():
    if "ctx" not in _keep:
        torch.cuda.init()
        torch.zeros(1, device="cuda")
        _keep["ctx"] = W.Context(0)
    return _keep["ctx"]


def _whir(params):
    w = _shared.get(params)
    if w is None:
        w = _shared[params] = W.Whir(_ctx(), *params)
    return w


def _server():
    s = _shared.get("server")
    if s is None:
        s = _shared["server"] = W.Server(workers=8)
    return s


class _Device(W.DeviceArray):
    """A torch tensor's memory as the package's device array."""

    def __init__(self, tensor):
        self.tensor = tensor
        self.ctx, self.ptr = _ctx(), tensor.data_ptr()
        self.nbytes = tensor.numel() * tensor.element_size()

    def close(self):
        self.ptr = None


def _words(gen, n, host=False):
    """n uniform field elements (Montgomery words), on the GPU or pinned on the host."""
    t = torch.randint(0, P, (int(n),), dtype=torch.int32, device="cuda", generator=gen)
    if not host:
        return t
    h = torch.empty(int(n), dtype=torch.int32, pin_memory=True)
    h.copy_(t)
    return h


def _host_words(gen, n):
    return _words(gen, n).cpu().numpy().view(np.uint32)


def _params(c):
    return (c["k"], c["folding"], c["rate"], c.get("initial_reduction", 1),
            c.get("soundness", JOHNSON), c.get("security", 100))


def _mix(c):
    """The jobs of a served mix: (k, rate, claims)."""
    r = random.Random(c["mix"])
    return [(r.randint(c["k_lo"], c["k_hi"]), r.randint(1, 2), r.randint(1, 4))
            for _ in range(c["jobs"])]


def _stacked_k(c):
    total = sum(1 << int(s) for s in c["sizes"].split(","))
    return (total - 1).bit_length()


def prepare(case, seed):
    c, kind = case, case["kind"]
    ctx = _ctx()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    s = {"case": c}
    if kind == "prove":
        t = _words(gen, 1 << c["k"], c["host"])
        s["poly"] = t.numpy().view(np.uint32) if c["host"] else _Device(t)
        s["hold"] = t
        s["whir"] = _whir(_params(c))
    elif kind == "stack":
        ks = [int(x) for x in c["sizes"].split(",")]
        s["ks"] = ks
        s["poly"] = _Device(_words(gen, sum(1 << k for k in ks)))
        s["whir"] = _whir((_stacked_k(c), c["folding"], c["rate"], 1, c["soundness"],
                           c["security"]))
        # every polynomial is claimed at a point shared by those of its size,
        # the largest ones twice
        sizes = sorted(set(ks), reverse=True)
        s["groups"] = [[i for i, k in enumerate(ks) if k == z] for z in sizes]
        s["groups"].append(s["groups"][0])
    elif kind == "batch":
        s["polys"] = [_Device(_words(gen, 1 << c["k"])) for _ in range(c["n"])]
    elif kind == "serve":
        s["server"] = _server()
        s["polys"] = [_words(gen, 1 << k, True) for k, _, _ in _mix(c)]
    elif kind == "verify":
        polys = [_Device(_words(gen, 1 << c["k"])) for _ in range(c["n"])]
        torch.cuda.synchronize()
        s["proofs"] = [p for p, _ in W.prove_batch(ctx, _params(c), polys, claims=c["claims"])]
        s["proofs"][0] = _corrupt(s["proofs"][0], seed)
    elif kind == "merkle":
        s["rows"] = _Device(_words(gen, c["row_len"] << c["log_h"]))
        r = random.Random(seed)
        s["idx"] = [r.randrange(1 << c["log_h"]) for _ in range(c["openings"])]
    elif kind == "dft":
        s["in"] = _words(gen, c["h_in"] * c["width"])
        s["out"] = torch.empty(c["width"] << c["log_h"], dtype=torch.int32, device="cuda")
    else:
        k, kept = c["k"], c["kept"]
        n = 1 << (k - kept)
        s["poly"] = _words(gen, 1 << k)
        s["point"] = _host_words(gen, 4 * k)
        s["eqs"] = _host_words(gen, 4 * (k - kept) * c["eqs"])
        s["vars"] = _host_words(gen, c["pows"])
        s["alpha"], s["r"] = _host_words(gen, 4), _host_words(gen, 4 * kept)
        s["p"] = [torch.empty(4 * (n >> i), dtype=torch.int32, device="cuda")
                  for i in range(kept + 1)]
        s["w"] = [torch.empty_like(t) for t in s["p"]]
    torch.cuda.synchronize()
    return s


def _corrupt(proof, seed):
    """One proof of a batch arrives damaged, as a verifier has to expect."""
    b = bytearray(proof)
    b[random.Random(seed).randrange(len(b))] ^= 1
    return bytes(b)


# ---------------------------------------------------------------- one pass
def _u32(a):
    return a.ctypes.data_as(W.u32p)


def _sized(data, bound):
    """Proof bytes in a buffer of their upper bound (a proof's length varies with
    the queries that coincide); only the part written is touched."""
    out = np.zeros(bound, np.uint8)
    out[:len(data)] = np.frombuffer(data, np.uint8)
    return out


def _proof_out(t, params, claims):
    cp = t.draw_base()
    data = t.finalize()
    return {"proof": _sized(data, W.proof_bound(params, claims)), "length": len(data),
            "checkpoint": cp}


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    ctx = _ctx()
    if kind == "prove":
        t = W.PoseidonWriter()
        state["whir"].prove(t, state["poly"], [c["k"]], [[0]] * c["claims"])
        return _proof_out(t, _params(c), c["claims"])
    if kind == "stack":
        t = W.PoseidonWriter()
        state["whir"].prove(t, state["poly"], state["ks"], state["groups"])
        return _proof_out(t, state["whir"].params, sum(len(g) for g in state["groups"]))
    if kind == "batch":
        got = W.prove_batch(ctx, _params(c), state["polys"], claims=c["claims"],
                            commit_only=c["commit_only"])
        bound = 64 if c["commit_only"] else W.proof_bound(_params(c), c["claims"])
        return _joined([p for p, _ in got], [cp for _, cp in got], bound * c["n"])
    if kind == "serve":
        jobs = [W.Job((k, 4, rate, 1, JOHNSON, 100), t.numpy().view(np.uint32), claims=claims)
                for (k, rate, claims), t in zip(_mix(c), state["polys"])]
        state["server"].run(jobs)
        bound = sum(W.proof_bound(j.params, j.claims) for j in jobs)
        return _joined([j.proof for j in jobs], [j.checkpoint for j in jobs], bound)
    if kind == "verify":
        got = W.verify_batch(ctx, _params(c), [c["k"]], [[0]] * c["claims"], state["proofs"])
        return np.array(got, np.int64)
    if kind == "merkle":
        tree = W.MerkleTree(ctx, state["rows"], c["log_h"], c["row_len"])
        opened = tree.open(state["idx"])
        tree.close()
        return {"root": tree.root, "opened": opened}
    lib = W.lib()
    if kind == "dft":
        W._check(lib.whir_dft_batch(ctx.h, state["in"].data_ptr(), c["h_in"], c["width"],
                                    c["log_h"], state["out"].data_ptr()))
        return state["out"]
    return _pieces(state, lib, ctx.h)


def _joined(proofs, checkpoints, bound):
    return {"proofs": _sized(b"".join(proofs), bound),
            "lengths": np.array([len(p) for p in proofs], np.int64),
            "checkpoints": np.array(checkpoints, np.int64)}


def _pieces(s, lib, h):
    """One claim (high variables fixed), the expression at the low variables'
    challenges, its constraint weights, and `kept` sumcheck rounds."""
    c = s["case"]
    k, kept = c["k"], c["kept"]
    n, pt, rs = k - kept, s["point"], s["r"]
    claim = np.empty(4 << kept, np.uint32)
    p, w = s["p"], s["w"]
    check = W._check
    check(lib.whir_compress_hi(h, s["poly"].data_ptr(), k, _u32(pt[4 * kept:]), n, _u32(claim)))
    check(lib.whir_compress_lo(h, s["poly"].data_ptr(), k, _u32(rs), kept, p[0].data_ptr()))
    check(lib.whir_eq_table(h, _u32(pt[4 * kept:]), n, _u32(s["alpha"]), w[0].data_ptr()))
    check(lib.whir_combine_eqs(h, w[0].data_ptr(), n, _u32(s["eqs"]), c["eqs"],
                               _u32(s["alpha"])))
    check(lib.whir_combine_pows(h, w[0].data_ptr(), n, _u32(s["vars"]), c["pows"],
                                _u32(s["alpha"]), c["eqs"]))
    ev = np.empty(4, np.uint32)
    check(lib.whir_eval_ext(h, p[0].data_ptr(), n, _u32(pt[4 * kept:]), _u32(ev)))
    rounds = []
    for i in range(kept):
        c0, c2 = np.empty(4, np.uint32), np.empty(4, np.uint32)
        check(lib.whir_sumcheck_coeffs(h, p[i].data_ptr(), w[i].data_ptr(), n - i, _u32(c0),
                                       _u32(c2)))
        check(lib.whir_sumcheck_fold(h, p[i].data_ptr(), w[i].data_ptr(), n - i,
                                     _u32(rs[4 * i:]), p[i + 1].data_ptr(),
                                     w[i + 1].data_ptr()))
        rounds += [c0, c2]
    return {"claim": claim, "eval": ev, "rounds": np.concatenate(rounds), "poly": p[kept],
            "weights": w[kept]}


# ---------------------------------------------------------------- what a pass cannot do without
def _perm_ops(width):
    """Field operations of one Poseidon2 permutation: two products per S-box,
    the light layers' adds, the internal layers' sum and scaled add."""
    rp = 20 if width == 16 else 23
    return 2 * (8 * width + rp) + 9 * 5 * width + rp * 3 * width


def _commit_ops(log_h, row_words, log_in):
    rows = 1 << log_h
    leaf = rows * -(-row_words // 16) * _perm_ops(24)
    tree = (rows - 1) * _perm_ops(16)
    dft = rows * row_words * 1.5 * max(1, log_in)
    return leaf + tree + dft


def _prove_ops(k, folding, rate, claims, commit_only=False):
    ops = _commit_ops(k + rate - folding, 1 << folding, k - folding)
    if commit_only:
        return ops
    n_rounds = max(0, -(-(k - 6) // folding) - 1) if k > 6 else 0
    for r in range(n_rounds):
        kp = k - folding * (r + 1)
        this = rate + (r + 1) * (folding - 1)
        ops += _commit_ops(kp + this - folding, 4 << folding, kp - folding)
    ext = 28  # field operations of one extension product
    return ops + (claims + 2) * 8 * (1 << k) + 8 * ext * (2 << (k - folding))


def work(case):
    c, kind = case, case["kind"]
    if kind == "prove":
        proof = 16384 + 4096 * c["k"]
        return {"bytes": 4 * (1 << c["k"]) + proof,
                "flops": _prove_ops(c["k"], c["folding"], c["rate"], c["claims"])}
    if kind == "stack":
        k, n = _stacked_k(c), sum(1 << int(x) for x in c["sizes"].split(","))
        return {"bytes": 4 * n + 16384 + 4096 * k,
                "flops": _prove_ops(k, c["folding"], c["rate"], len(c["sizes"].split(",")))}
    if kind == "batch":
        return {"bytes": c["n"] * (4 << c["k"]),
                "flops": c["n"] * _prove_ops(c["k"], c["folding"], c["rate"], c["claims"],
                                             c["commit_only"])}
    if kind == "serve":
        jobs = _mix(c)
        return {"bytes": sum(4 << k for k, _, _ in jobs),
                "flops": sum(_prove_ops(k, 4, rate, claims) for k, rate, claims in jobs)}
    if kind == "verify":
        log_h = c["k"] + c["rate"] - c["folding"]
        opened = 150 * c["n"]
        return {"bytes": opened * 4 * ((2 << c["folding"]) + 8 * log_h),
                "flops": opened * (_perm_ops(24) * 2 + log_h * _perm_ops(16))}
    if kind == "merkle":
        rows = 1 << c["log_h"]
        return {"bytes": 4 * rows * c["row_len"],
                "flops": rows * (-(-c["row_len"] // 16) * _perm_ops(24) + _perm_ops(16))}
    if kind == "dft":
        words = c["width"] << c["log_h"]
        return {"bytes": 4 * (c["h_in"] * c["width"] + words),
                "flops": words * 1.5 * max(1, (c["h_in"] - 1).bit_length())}
    n = 1 << (c["k"] - c["kept"])
    return {"bytes": 8 * (1 << c["k"]) + 16 * n * 12,
            "flops": 16.0 * (1 << c["k"]) + n * (28 * (c["eqs"] + 12) + 8 * c["pows"])}


def exact(case, seed):
    """Every output is a field element, a digest, an index or proof bytes: whole
    numbers, which have to be equal, so there is no rounding to measure."""
    return None
