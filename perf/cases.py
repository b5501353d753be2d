"""Performance cases: the operations a program has this library do, on data that already lives on the GPU.

Tensors are flat torch buffers in the library's layout (dense, column-major: dimension 0 is the fastest), handed to
the public entry points of `tal_sh_b200`: the TAL-SH C API (`talshTensorContract`, `talshTensorAdd`) for the small
drop-in calls, the device ABI (`tc*`) for everything else.  Offset-table scratch is queried and allocated once per
shape, as the library's callers do.  `exact` repeats a case in 64-bit torch.
"""
import ctypes as C
import math
import re

import torch

import tal_sh_b200 as T

KINDS = {"r4": T.R4, "r8": T.R8, "c4": T.C4, "c8": T.C8}
DTYPE = {"r4": torch.float32, "r8": torch.float64, "c4": torch.complex64, "c8": torch.complex128}
ESIZE = {"r4": 4, "r8": 8, "c4": 8, "c8": 16}
MAX_ELEMS = 1 << 27  # of one tensor of a drawn contraction

# Contractions of coupled-cluster codes with a large output: ladders, rings and one-index transformations.
DENSE = ["D(a,b,i,j)+=L(a,k,c,i)*R(c,b,k,j)", "D(a,b,i,j)+=L(a,b,c,d)*R(c,d,i,j)",
         "D(a,b,c,d)+=L(a,e,b,f)*R(d,f,c,e)", "D(a,b,c,d)+=L(e,a,f,c)*R(b,f,d,e)",
         "D(a,b,c)+=L(a,d,e,c)*R(e,b,d)", "D(a,b,c,d)+=L(e,b,a,d)*R(c,e)",
         "D(a,b,c,d)+=L(e,c)*R(a,b,e,d)", "D(a,b)+=L(c,a,d)*R(d,c,b)",
         "D(a,b,c,d,e,f)+=L(d,e,g,a)*R(g,f,b,c)"]
# Intermediates: a small output and a long contracted range (the one-body F and W tensors, densities).
SMALL_OUT = ["D(m,i)+=L(m,k,c,d)*R(i,k,c,d)", "D(a,e)+=L(k,c,a,l)*R(l,c,k,e)", "D(m,e)+=L(m,k,e,c)*R(c,k)",
             "D(i)+=L(i,j,k)*R(k,j)", "D(a,i)+=L(a,c,k,d)*R(c,d,k,i)"]
# Full contractions: energies and overlaps of two amplitude tensors, stored alike or not.
FULL = ["D()+=L(a,b,i,j)*R(a,b,i,j)", "D()+=L(a,b,i,j)*R(b,a,i,j)", "D()+=L(a,b,i,j)*R(i,j,a,b)"]


def listed():
    return [
        # The smallest calls: the drop-in API on tiny GPU-resident tensors, where launches and host work are all.
        dict(name="small_calls", op="small", kind="r8", v=13, o=12),
        # Index reorderings before and after other codes' kernels: double precision, ordinary rank, large.
        dict(name="transpose_r8", op="copy", kind="r8", dims="279,37,196,31", perm="3,1,4,2"),
        # The same in single precision with odd extents and higher rank, where no run is aligned.
        dict(name="transpose_r4_odd", op="copy", kind="r4", dims="31,17,97,11,45", perm="4,2,5,1,3"),
        # Residual update with a permuted tensor (antisymmetriser term), single precision, odd extents.
        dict(name="transpose_add_r4", op="add", kind="r4", dims="97,41,83,67", perm="2,4,1,3"),
        # The coupled-cluster ring contraction at its full size (v = 96, o = 32), double precision.
        dict(name="contract_r8_ring", op="contract", kind="r8", pattern=DENSE[0],
             ext="a=96,b=96,c=96,i=32,j=32,k=32"),
        # A single-precision ladder of ordinary size.
        dict(name="contract_r4", op="contract", kind="r4", pattern=DENSE[1], ext="a=57,b=57,c=57,d=57,i=24,j=24"),
        # Complex double precision with a conjugated operand, odd extents (relativistic and response codes).
        dict(name="contract_c8_odd", op="contract", kind="c8", pattern="D(a,b,c,d)+=L+(a,e,b,f)*R(d,f,c,e)",
             ext="a=37,b=31,c=29,d=33,e=35,f=27"),
        # One-body intermediate: 40 x 40 outputs, a contracted range of half a million.
        dict(name="intermediate_r8", op="contract", kind="r8", pattern=SMALL_OUT[0], ext="m=40,i=40,k=40,c=112,d=112"),
        # Energy: full contraction of two amplitude tensors stored in different index orders.
        dict(name="energy_r8", op="contract", kind="r8", pattern=FULL[1], ext="a=112,b=112,i=40,j=40"),
        # Many independent small contractions in one call (block-sparse codes): ranks 2-6, extents 4-48, R8 and C8.
        dict(name="batch_mixed", op="batch", ntasks=768, emax=48, shapes=11),
        # The ring contraction through the int8 split form (1e-11 relative error) with odd extents.
        dict(name="split_int8", op="split", kind="r8", pattern=DENSE[0], ext="a=88,b=85,c=80,i=30,j=33,k=31"),
        # Blocked algorithms: cut a block out, scale it, add it into another tensor, take its norm.
        dict(name="block_update_r8", op="block", kind="r8", dims="97,61,75,83", block="71,44,53,60",
             offs="13,9,17,20"),
    ]


# ----------------------------------------------------------------------------------------------------- drawing
def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _odd(rng, x):
    """x, or one of its odd neighbours."""
    x = max(2, int(round(x)))
    return x if rng.random() < 0.5 else x | 1


def _text(xs):
    return ",".join(str(int(x)) for x in xs)


def _draw_dims(rng, rank, lo, hi):
    """Extents of one tensor of rank `rank` with lo..hi elements."""
    while True:
        vol = _log(rng, lo, hi)
        w = [rng.gammavariate(1.5, 1.0) for _ in range(rank)]
        dims = [_odd(rng, vol ** (x / sum(w))) for x in w]
        if lo <= math.prod(dims) <= hi:
            return dims


def _draw_contraction(rng, patterns, flop_lo, flop_hi, kind, spread):
    while True:
        pattern = rng.choice(patterns)
        d, l, r = _labels(pattern)
        names = sorted(set(l + r))
        free = _log(rng, flop_lo, flop_hi) / (8 if kind[0] == "c" else 2)
        w = {x: math.exp(rng.uniform(-spread, spread)) for x in names}
        base = (free / math.prod(w.values())) ** (1.0 / len(names))
        ext = {x: _odd(rng, base * w[x]) for x in names}
        flops = math.prod(ext.values()) * (8 if kind[0] == "c" else 2)
        big = max(math.prod(ext[x] for x in t) for t in (d, l, r))
        if big <= MAX_ELEMS and flop_lo <= flops <= flop_hi:
            return dict(op="contract", kind=kind, pattern=pattern, ext=",".join("%s=%d" % (x, ext[x]) for x in names))


def draw(rng):
    op = rng.choice(["small", "copy", "copy", "add", "dense", "dense", "dense", "small_out", "full", "batch", "split",
                     "block"])
    if op == "small":
        return dict(op="small", kind=rng.choice(["r4", "r8", "c8"]), v=rng.randint(4, 20), o=rng.randint(3, 16))
    if op in ("copy", "add"):
        rank = rng.randint(2, 6)
        dims = _draw_dims(rng, rank, 1 << 14, 1 << 27)
        perm = list(range(1, rank + 1))
        while perm == sorted(perm):
            rng.shuffle(perm)
        return dict(op=op, kind=rng.choice(["r4", "r4", "r8", "r8", "c8"]), dims=_text(dims), perm=_text(perm))
    if op == "dense":
        kind = rng.choice(["r8", "r8", "r4", "r4", "c8", "c4"])
        return _draw_contraction(rng, DENSE, 2e7, 1.5e11, kind, 0.5)
    if op == "small_out":
        return _draw_contraction(rng, SMALL_OUT, 1e7, 1e10, rng.choice(["r8", "r8", "r4", "c8"]), 0.4)
    if op == "full":
        return _draw_contraction(rng, FULL, 1e5, 1.5e8, rng.choice(["r8", "r4", "c8"]), 0.4)
    if op == "batch":
        return dict(op="batch", ntasks=int(_log(rng, 32, 768)), emax=rng.randint(12, 48), shapes=rng.randint(1, 1 << 20))
    if op == "split":
        c = _draw_contraction(rng, DENSE[:4], 2e9, 1.5e11, "r8", 0.4)
        c["op"] = "split"
        return c
    rank = rng.randint(2, 5)
    dims = _draw_dims(rng, rank, 1 << 14, 1 << 26)
    block = [rng.randint(max(1, x // 3), x) for x in dims]
    offs = [rng.randint(0, x - y) for x, y in zip(dims, block)]
    return dict(op="block", kind=rng.choice(["r4", "r8", "c8"]), dims=_text(dims), block=_text(block), offs=_text(offs))


# ------------------------------------------------------------------------------------------------- case contents
def _ints(text):
    return [int(x) for x in text.split(",")]


def _ext(case):
    return {x.split("=")[0]: int(x.split("=")[1]) for x in case["ext"].split(",")}


def _labels(pattern):
    """Index labels of D, L, R (or D, L) in a symbolic pattern."""
    return [[x for x in g.split(",") if x] for g in re.findall(r"\(([a-z,]*)\)", pattern)]


def _vol(dims):
    return math.prod(dims) if dims else 1


def _rand(gen, n, kind):
    """n values uniform in [-1, 1) (complex: both parts)."""
    real = {"r4": torch.float32, "c4": torch.float32}.get(kind, torch.float64)
    x = torch.rand(n * (2 if kind[0] == "c" else 1), dtype=real, device="cuda", generator=gen).mul_(2.0).sub_(1.0)
    return torch.view_as_complex(x.view(n, 2)) if kind[0] == "c" else x


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _check(rc, what):
    if rc != 0:
        raise RuntimeError("%s failed: %d (%s)" % (what, rc, T.lib().tcLastErrorString()))


_started = False


def _talsh():
    """The library with TAL-SH started on GPU 0."""
    global _started
    lib = T.lib()
    if not _started:
        host, args = C.c_size_t(0), C.c_int(0)
        _check(lib.talshInit(C.byref(host), C.byref(args), 1, T.ivec([0]), 0, None, 0, None), "talshInit")
        _started = True
    return lib


class _Attached:
    """A TAL-SH tensor whose body is a torch buffer on GPU 0."""

    def __init__(self, lib, buf, dims, kind):
        self.lib, self.buf, self.t = lib, buf, T.Tens()
        _check(lib.talshTensorClean(C.byref(self.t)), "talshTensorClean")
        _check(lib.talshTensorConstruct(C.byref(self.t), KINDS[kind], len(dims), T.ivec(dims),
                                        lib.talshFlatDevId(T.DEV_NVIDIA_GPU, 0), buf.data_ptr(), -1, None, 0.0, 0.0),
               "talshTensorConstruct")
        self.ref = C.byref(self.t)

    def __del__(self):
        self.lib.talshTensorDestruct(C.byref(self.t))


SMALL_CONTRACT = "D(a,b,i,j)+=L(a,k,c,i)*R(c,b,k,j)"
SMALL_ADD = "D(b,a,j,i)+=L(a,b,i,j)"


def _batch_tasks(case):
    """Shapes of a batch's tasks: operand ranks 2-6, 1-3 contracted indices, extents log-uniform in [4, emax]."""
    import random
    rng = random.Random(case["shapes"])
    out = []
    while len(out) < case["ntasks"]:
        nc = rng.randint(1, 3)
        lu, ru = rng.randint(max(2, nc), 6) - nc, rng.randint(max(2, nc), 6) - nc
        ext = [int(round(_log(rng, 4, case["emax"]))) for _ in range(nc + lu + ru)]
        c, lo, ro = list(range(nc)), list(range(nc, nc + lu)), list(range(nc + lu, nc + lu + ru))
        li, ri, di = c + lo, c + ro, lo + ro
        for x in (li, ri, di):
            rng.shuffle(x)
        if max(_vol([ext[i] for i in x]) for x in (li, ri, di)) > 1 << 21:
            continue
        out.append(("r8" if len(out) % 2 == 0 else "c8", [[ext[i] for i in x] for x in (di, li, ri)], (di, li, ri)))
    return out


def _contract_shapes(case):
    d, l, r = _labels(case["pattern"])
    e = _ext(case)
    return [[e[x] for x in t] for t in (d, l, r)]


def _alpha(case):
    return (0.5, -0.25) if case["kind"][0] == "c" else (0.5, 0.0)


def _contract_buffers(case, seed):
    g = _gen(seed)
    return [_rand(g, _vol(x), case["kind"]) for x in _contract_shapes(case)]


def _block_buffers(case, seed):
    g, k = _gen(seed), case["kind"]
    full, target = (_rand(g, _vol(_ints(case["dims"])), k) for _ in range(2))
    return full, target


def _batch_buffers(case, seed):
    """Per kind, one buffer with every task's operands and one zeroed buffer for the results, and where each task's
    L, R and D start in them (elements)."""
    g, pad = _gen(seed), lambda dims: (_vol(dims) + 31) // 32 * 32  # noqa: E731
    at, out_at, places = {"r8": 0, "c8": 0}, {"r8": 0, "c8": 0}, []
    for kind, (dd, ld, rd), idx in _batch_tasks(case):
        places.append((kind, dd, ld, rd, idx, at[kind], at[kind] + pad(ld), out_at[kind]))
        at[kind] += pad(ld) + pad(rd)
        out_at[kind] += pad(dd)
    ins = {k: _rand(g, max(at[k], 32), k) for k in ("r8", "c8")}
    outs = {k: torch.zeros(max(out_at[k], 32), dtype=DTYPE[k], device="cuda") for k in ("r8", "c8")}
    return ins, outs, places


def prepare(case, seed):
    lib, op = T.lib(), case["op"]
    s = dict(op=op, lib=lib)
    if op == "small":
        lib = s["lib"] = _talsh()
        g, k, v, o = _gen(seed), case["kind"], case["v"], case["o"]
        shapes = dict(t=[v, v, o, o], l=[v, o, v, o], r=[v, v, o, o], d=[v, v, o, o])
        s["buf"] = {x: _rand(g, _vol(shapes[x]), k) for x in shapes}
        torch.cuda.synchronize()
        s["tens"] = {x: _Attached(lib, s["buf"][x], shapes[x], k) for x in shapes}
    elif op in ("copy", "add"):
        g, k, dims = _gen(seed), case["kind"], _ints(case["dims"])
        s["src"] = _rand(g, _vol(dims), k)
        s["dst"] = _rand(g, _vol(dims), k) if op == "add" else torch.zeros_like(s["src"])
        s["args"] = (KINDS[k], len(dims), T.ivec(dims), T.ivec(_ints(case["perm"])))
        s["alpha"] = _alpha(case)
    elif op in ("contract", "split"):
        k = case["kind"]
        s["d"], s["l"], s["r"] = _contract_buffers(case, seed)
        dd, ld, rd = _contract_shapes(case)
        rc, dig, dr, lr, rr, conj = T.parse_pattern(case["pattern"])
        _check(rc, "pattern")
        s["args"] = (KINDS[k], T.ivec(dig), dr, T.ivec(dd), lr, T.ivec(ld), rr, T.ivec(rd))
        s["alpha"], s["conj"] = _alpha(case), conj
        if op == "split":
            need = lib.tcTensorContractSplitScratch(*s["args"], 6)
        else:
            need = lib.tcTensorContractScratch(*s["args"])
        s["scratch"] = torch.empty(max(need, 16), dtype=torch.uint8, device="cuda")
        s["need"] = need
    elif op == "batch":
        s["ins"], s["outs"], places = _batch_buffers(case, seed)
        arr = (T.ContractTask * len(places))()
        for t, (kind, dd, ld, rd, (di, li, ri), at_l, at_r, at_d) in zip(arr, places):
            t.data_kind, t.drank, t.lrank, t.rrank = KINDS[kind], len(dd), len(ld), len(rd)
            for i, x in enumerate(li):
                t.cptrn[i] = di.index(x) + 1 if x in di else -(ri.index(x) + 1)
            for i, x in enumerate(ri):
                t.cptrn[len(li) + i] = di.index(x) + 1 if x in di else -(li.index(x) + 1)
            for to, dims in ((t.ddims, dd), (t.ldims, ld), (t.rdims, rd)):
                for i, x in enumerate(dims):
                    to[i] = x
            t.L, t.R = (s["ins"][kind].data_ptr() + x * ESIZE[kind] for x in (at_l, at_r))
            t.D = s["outs"][kind].data_ptr() + at_d * ESIZE[kind]
            t.alpha_re, t.alpha_im, t.conj_bits, t.accumulative = 1.0, 0.0, 0, 1
        s["tasks"] = arr
        s["need"] = lib.tcTensorContractBatchScratch(len(arr), arr)
        s["scratch"] = torch.empty(s["need"], dtype=torch.uint8, device="cuda")
    else:
        k, dims, block = case["kind"], _ints(case["dims"]), _ints(case["block"])
        s["full"], s["target"] = _block_buffers(case, seed)
        s["block"] = torch.empty(_vol(block), dtype=DTYPE[k], device="cuda")
        s["args"] = (KINDS[k], len(dims), T.ivec(dims), T.ivec(block), T.ivec(_ints(case["offs"])))
        s["norm"] = torch.zeros(1, dtype=torch.float64, device="cuda")
        s["need"] = lib.tcTensorNorm1Scratch(_vol(block))
        s["scratch"] = torch.empty(s["need"], dtype=torch.uint8, device="cuda")
        s["alpha"] = _alpha(case)
    return s


def run(s):
    lib, op = s["lib"], s["op"]
    if op == "small":  # blocking drop-in calls: T = L * R, then D += permuted T
        t = s["tens"]
        _check(lib.talshTensorContract(SMALL_CONTRACT.encode(), t["t"].ref, t["l"].ref, t["r"].ref, 1.0, 0.0, 0,
                                       T.DEV_NVIDIA_GPU, T.COPY_KKK, T.NOPE, None), "talshTensorContract")
        _check(lib.talshTensorAdd(SMALL_ADD.encode(), t["d"].ref, t["t"].ref, 0.5, 0.0, 0, T.DEV_NVIDIA_GPU,
                                  T.COPY_KK, None), "talshTensorAdd")
        return s["buf"]["t"], s["buf"]["d"]
    if op == "copy":
        _check(lib.tcTensorPermute(*s["args"], s["src"].data_ptr(), s["dst"].data_ptr(), 0, _stream()),
               "tcTensorPermute")
        return s["dst"]
    if op == "add":
        _check(lib.tcTensorPermuteAdd(*s["args"], s["src"].data_ptr(), s["dst"].data_ptr(), *s["alpha"], 0, _stream()),
               "tcTensorPermuteAdd")
        return s["dst"]
    if op == "contract":
        _check(lib.tcTensorContract(*s["args"], s["d"].data_ptr(), s["l"].data_ptr(), s["r"].data_ptr(), *s["alpha"],
                                    s["conj"], 1, s["scratch"].data_ptr(), s["need"], _stream()), "tcTensorContract")
        return s["d"]
    if op == "split":
        _check(lib.tcTensorContractSplit(*s["args"], s["d"].data_ptr(), s["l"].data_ptr(), s["r"].data_ptr(),
                                         *s["alpha"], s["conj"], 1, 6, s["scratch"].data_ptr(), s["need"], _stream()),
               "tcTensorContractSplit")
        return s["d"]
    if op == "batch":
        _check(lib.tcTensorContractBatch(len(s["tasks"]), s["tasks"], s["scratch"].data_ptr(), s["need"], _stream()),
               "tcTensorContractBatch")
        return s["outs"]["r8"], s["outs"]["c8"]
    kind, n, st = s["args"][0], s["block"].numel(), _stream()
    _check(lib.tcTensorSlice(*s["args"], s["full"].data_ptr(), s["block"].data_ptr(), 0, st), "tcTensorSlice")
    _check(lib.tcTensorScale(kind, n, s["block"].data_ptr(), *s["alpha"], st), "tcTensorScale")
    _check(lib.tcTensorInsert(*s["args"], s["block"].data_ptr(), s["target"].data_ptr(), 1, st), "tcTensorInsert")
    _check(lib.tcTensorNorm1(kind, n, s["block"].data_ptr(), s["norm"].data_ptr(), s["scratch"].data_ptr(), s["need"],
                             st), "tcTensorNorm1")
    return s["block"], s["target"], s["norm"]


def work(case):
    op = case["op"]
    if op == "small":
        v, o, es = case["v"], case["o"], ESIZE[case["kind"]]
        f = 8 if case["kind"][0] == "c" else 2
        n = v * v * o * o
        return dict(bytes=6 * n * es, flops=f * n * v * o + f * n)  # read L, R; write T; read T, D; write D
    if op in ("copy", "add"):
        n = _vol(_ints(case["dims"]))
        return dict(bytes=(3 if op == "add" else 2) * n * ESIZE[case["kind"]], flops=2 * n if op == "add" else 0)
    if op in ("contract", "split"):
        dd, ld, rd = _contract_shapes(case)
        f = 8 if case["kind"][0] == "c" else 2
        return dict(bytes=(2 * _vol(dd) + _vol(ld) + _vol(rd)) * ESIZE[case["kind"]],
                    flops=f * math.prod(_ext(case).values()))
    if op == "batch":
        b = f = 0
        for kind, (dd, ld, rd), (di, li, ri) in _batch_tasks(case):
            ext = {x: e for i, t in ((li, ld), (ri, rd)) for x, e in zip(i, t)}
            b += (2 * _vol(dd) + _vol(ld) + _vol(rd)) * ESIZE[kind]
            f += (8 if kind == "c8" else 2) * math.prod(ext.values())
        return dict(bytes=b, flops=f)
    n = _vol(_ints(case["block"])) * ESIZE[case["kind"]]
    return dict(bytes=(2 + 2 + 3 + 1) * n, flops=0)  # slice, scale, insert with addition, norm: one call each


# ------------------------------------------------------------------------------------------------------- checks
def _wide(x):
    return x.to(torch.complex128) if x.is_complex() else x.to(torch.float64)


def _cols(x, dims):
    """A column-major body as a torch view with the dimensions in reverse order."""
    return _wide(x).view(list(reversed(dims))) if dims else _wide(x).view(())


def _einsum(out, l, ldims, r, rdims, li, ri):
    """Column-major flat contraction of L[li] and R[ri] into the index order `out` (labels), in 64 bits."""
    names = {x: n for n, x in enumerate(dict.fromkeys(list(li) + list(ri)))}
    num = lambda idx: [names[x] for x in reversed(idx)]  # noqa: E731
    return torch.einsum(_cols(l, ldims), num(li), _cols(r, rdims), num(ri), num(out)).reshape(-1)


def exact(case, seed):
    op = case["op"]
    if op == "small":
        g, k, v, o = _gen(seed), case["kind"], case["v"], case["o"]
        _, l, r, d = (_rand(g, v * v * o * o, k) for _ in range(4))
        t = _einsum("abij", l, [v, o, v, o], r, [v, v, o, o], "akci", "cbkj")
        back = t.view(o, o, v, v).permute(1, 0, 3, 2).reshape(-1)  # T(a,b,i,j) -> D(b,a,j,i)
        return t, _wide(d) + 0.5 * back
    if op in ("copy", "add"):
        g, k, dims = _gen(seed), case["kind"], _ints(case["dims"])
        n2o = [0] * len(dims)
        for i, p in enumerate(_ints(case["perm"])):
            n2o[p - 1] = i
        rank = len(dims)
        src = _rand(g, _vol(dims), k)
        out = _cols(src, dims).permute([rank - 1 - n2o[rank - 1 - j] for j in range(rank)]).reshape(-1)
        if op == "copy":
            return out
        return _wide(_rand(g, _vol(dims), k)) + out * complex(*_alpha(case)) if k[0] == "c" else \
            _wide(_rand(g, _vol(dims), k)) + out * _alpha(case)[0]
    if op in ("contract", "split"):
        d, l, r = _contract_buffers(case, seed)
        di, li, ri = _labels(case["pattern"])
        dd, ld, rd = _contract_shapes(case)
        if "L+" in case["pattern"]:
            l = l.conj().resolve_conj()
        if not di:
            a = _cols(l, ld)
            b = _cols(r, rd).permute([list(reversed(ri)).index(x) for x in reversed(li)])
            out = (a * b).sum().view(1)
        else:
            out = _einsum(di, l, ld, r, rd, li, ri)
        a = complex(*_alpha(case)) if case["kind"][0] == "c" else _alpha(case)[0]
        return _wide(d) + a * out
    if op == "batch":
        ins, outs, places = _batch_buffers(case, seed)
        for kind, dd, ld, rd, (di, li, ri), at_l, at_r, at_d in places:
            l, r = ins[kind][at_l:at_l + _vol(ld)], ins[kind][at_r:at_r + _vol(rd)]
            outs[kind][at_d:at_d + _vol(dd)] += _einsum(di, l, ld, r, rd, li, ri)
        return outs["r8"], outs["c8"]
    full, target = _block_buffers(case, seed)
    dims, block, offs = _ints(case["dims"]), _ints(case["block"]), _ints(case["offs"])
    where = tuple(slice(o, o + b) for o, b in zip(reversed(offs), reversed(block)))
    a = complex(*_alpha(case)) if case["kind"][0] == "c" else _alpha(case)[0]
    part = _cols(full, dims)[where] * a
    out = _cols(target, dims).clone()
    out[where] += part
    return part.reshape(-1).contiguous(), out.reshape(-1), part.abs().sum().view(1)
