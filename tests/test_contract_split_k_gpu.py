"""Contractions whose contracted range is split over CTAs (few output tiles, long K): against numpy in 64 bits at
the edges of the split and of the tiles, equal bit for bit alone, repeated, in a batch, in a replayed graph and with a
scratch that has no room for the partial sums."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

import tal_sh_b200 as T
from gpu_util import rand, rel_err

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

TOL = {T.R8: 1e-12, T.C8: 1e-12, T.R4: 2e-5, T.C4: 2e-5}  # the parity bars of every contraction test
# (M, N, K): one tile and a remainder each way, K below / at / above two chunks, two-level sums, vectors
SHAPES = [(1, 1, 511), (1, 1, 513), (7, 9, 512), (32, 33, 1023), (40, 40, 20001), (64, 64, 769), (65, 1, 4097),
          (1, 130, 5000), (100, 70, 3000), (200, 150, 1600)]


def _launch(lib, torch, kind, dims, d, l, r, acc, conj=0, scratch=None, shift=0):
    m, n, k = dims
    args = (kind, T.ivec([-2, 1, 2, -1]), 2, T.ivec([m, n]), 2, T.ivec([k, m]), 2, T.ivec([n, k]))
    need = lib.tcTensorContractScratch(*args)
    size = need if scratch is None else scratch(need, m, n, k)
    buf = torch.empty(size + shift, dtype=torch.uint8, device="cuda")
    rc = lib.tcTensorContract(*args, d.data_ptr(), l.data_ptr(), r.data_ptr(), 0.5, 0.0, conj, acc,
                              buf.data_ptr() + shift, size, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return rc


@pytest.mark.parametrize("kind", [T.R8, T.C8, T.R4, T.C4])
def test_split_k_matches_numpy_alone_and_batched(talsh, kind):
    torch = pytest.importorskip("torch")
    lib, rng = T.lib(), np.random.default_rng(5)
    dev = lambda a: torch.from_numpy(np.asarray(a).ravel(order="F").copy()).cuda()
    tasks = (T.ContractTask * len(SHAPES))()
    keep, starts = [], []
    for t, (m, n, k) in zip(tasks, SHAPES):
        L, R, D0 = rand([k, m], kind, rng), rand([n, k], kind, rng), rand([m, n], kind, rng)
        conj = 0 if kind in (T.R4, T.R8) else 2  # conj(L)
        ref = D0.astype(np.complex128) + 0.5 * (np.conj(L.astype(np.complex128)).T @ R.astype(np.complex128).T)
        l, r, out = dev(L), dev(R), [dev(D0) for _ in range(7)]
        for d in out[:2]:
            assert _launch(lib, torch, kind, (m, n, k), d, l, r, 1, conj) == 0
        least = lambda need, m, n, k: (16 * (m + n + k) + 255) // 256 * 256  # the offset tables alone
        assert _launch(lib, torch, kind, (m, n, k), out[2], l, r, 1, conj, least) == 0
        assert _launch(lib, torch, kind, (m, n, k), out[6], l, r, 1, conj, shift=8) == 0  # partial sums want 16 bytes
        short = lambda need, m, n, k: least(need, m, n, k) - 256
        assert _launch(lib, torch, kind, (m, n, k), out[3], l, r, 1, conj, short) == T.TALSH_INVALID_ARGS
        for d in (out[1], out[2], out[6]):
            assert torch.equal(d, out[0]), (m, n, k)
        assert rel_err(out[0].cpu().numpy().reshape(ref.shape, order="F"), ref) <= TOL[kind], (m, n, k)
        t.data_kind, t.drank, t.lrank, t.rrank = kind, 2, 2, 2
        for i, v in enumerate([-2, 1, 2, -1]):
            t.cptrn[i] = v
        for to, dims in ((t.ddims, [m, n]), (t.ldims, [k, m]), (t.rdims, [n, k])):
            for i, v in enumerate(dims):
                to[i] = v
        t.D, t.L, t.R = out[3].data_ptr(), l.data_ptr(), r.data_ptr()
        t.alpha_re, t.alpha_im, t.conj_bits, t.accumulative = 0.5, 0.0, conj, 1
        keep.append((out, l, r))
        starts.append(dev(D0))
    need = lib.tcTensorContractBatchScratch(len(SHAPES), tasks)
    buf = torch.empty(need, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    # whole scratch; 256 bytes short (the batch has no partial sums); a graph of each, replayed
    for o, size in ((3, need), (4, need - 256)):
        for t, (out, _, _) in zip(tasks, keep):
            t.D = out[o].data_ptr()
        assert lib.tcTensorContractBatch(len(SHAPES), tasks, buf.data_ptr(), size, s) == 0
        torch.cuda.synchronize()
        for (out, _, _), dims in zip(keep, SHAPES):
            assert torch.equal(out[o], out[0]), dims
        for t, (out, _, _) in zip(tasks, keep):
            t.D, t.accumulative = out[5].data_ptr(), 0
        g = C.c_void_p()
        assert lib.tcContractBatchGraphCreate(len(SHAPES), tasks, buf.data_ptr(), size, s, C.byref(g)) == 0
        first = None
        for _ in range(3):
            for out, _, _ in keep:
                out[5].fill_(float("nan"))
            assert lib.tcContractBatchGraphLaunch(g, s) == 0
            torch.cuda.synchronize()
            got = [out[5].clone() for out, _, _ in keep]
            first = first or got
            assert all(torch.equal(a, b) for a, b in zip(got, first))
        assert lib.tcContractBatchGraphDestroy(g) == 0
        for x, (out, _, _), d0 in zip(first, keep, starts):  # 0.5 L R: the sums of the accumulating calls
            assert rel_err((d0 + x).cpu().numpy(), out[0].cpu().numpy()) <= TOL[kind]
        for t in tasks:
            t.accumulative = 1
    assert lib.tcTensorContractBatch(len(SHAPES), tasks, buf.data_ptr(), sum(16 * sum(x) for x in SHAPES),
                                     s) == T.TALSH_INVALID_ARGS  # the tables alone, no descriptors


def test_split_k_with_hyper_indices(talsh):
    """Hyper combinations times splits: D(a,h,b) = L(k,h,a) R(b,k,h), with the partial sums and without."""
    torch = pytest.importorskip("torch")
    lib, rng = T.lib(), np.random.default_rng(6)
    a, b, h, k = 33, 18, 5, 3001
    L, R = rand([k, h, a], T.R8, rng), rand([b, k, h], T.R8, rng)
    ref = np.einsum("kha,bkh->ahb", L, R)
    dev = lambda x: torch.from_numpy(np.asarray(x).ravel(order="F").copy()).cuda()
    d, d2, l, r = dev(np.zeros((a, h, b))), dev(np.zeros((a, h, b))), dev(L), dev(R)
    args = (T.R8, T.ivec([-2, 2, 1, 3, -1, 2]), 3, T.ivec([a, h, b]), 3, T.ivec([k, h, a]), 3, T.ivec([b, k, h]))
    need = lib.tcTensorContractScratch(*args)
    buf = torch.empty(need, dtype=torch.uint8, device="cuda")
    for out, size in ((d, need), (d2, need - 256)):
        assert lib.tcTensorContract(*args, out.data_ptr(), l.data_ptr(), r.data_ptr(), 1.0, 0.0, 0, 0, buf.data_ptr(),
                                    size, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert rel_err(d.cpu().numpy().reshape(ref.shape, order="F"), ref) <= TOL[T.R8]
    assert torch.equal(d, d2)


@pytest.mark.parametrize("kind,xl,dims", [(T.R8, 0, (40, 33, 20001)), (T.R4, 0, (40, 33, 20001)),
                                          (T.R4, 1, (1, 1, 230000))])
def test_short_device_memory_changes_no_bits(kind, xl, dims):
    """talshTensorContract and the out-of-core form in a pool that holds the operands and the offset tables but not
    the partial sums: the bits of a roomy pool, and no deferred task on record."""
    code = r"""
import ctypes as C, hashlib, sys
import numpy as np
sys.path.insert(0, %r)
import tal_sh_b200 as T
L = T.lib()
hb, ha = C.c_size_t(0), C.c_int(0)
assert L.talshInit(C.byref(hb), C.byref(ha), 1, T.ivec([0]), 0, None, 0, None) == 0
rng = np.random.default_rng(11)
kind, xl, (m, n, k) = %d, %d, %r
A, B = (np.asfortranarray(rng.uniform(-1, 1, x).astype(T.NP_DTYPE[kind])) for x in ([k, m], [n, k]))
D = np.asfortranarray(np.zeros((m, n), dtype=A.dtype))
t = [T.Tensor(list(x.shape), kind, 0, ext=x) for x in (D, A, B)]
args = (b"D(a,b)+=L(k,a)*R(b,k)", t[0].ref, t[1].ref, t[2].ref, 1.0, 0.0, 0, T.DEV_NVIDIA_GPU)
rc = L.talshTensorContractXL(*args, T.YEP) if xl else L.talshTensorContract(*args, T.COPY_TTT, T.YEP, None)
assert rc == 0, rc
assert not xl or L.tcContractXLLastOps() == 1
for x in t:
    assert x.destruct() == 0
print("sum", hashlib.sha256(D.tobytes()).hexdigest())
L.talshStats(0, T.DEV_NVIDIA_GPU)
assert L.talshShutdown() == 0
""" % (ROOT, kind, xl, dims)
    m, n, k = dims
    up = lambda b: (b + 255) // 256 * 256  # noqa: E731
    body = sum(up((8 if kind == T.R8 else 4) * x) for x in (m * n, m * k, n * k))
    # an out-of-core block takes at most a quarter of the pool
    short = 4 * body if xl else body + up(16 * (m + n + k))
    scratch = T.lib().tcTensorContractScratch(kind, T.ivec([-2, 1, 2, -1]), 2, T.ivec([m, n]), 2, T.ivec([k, m]), 2,
                                              T.ivec([n, k]))
    assert short + 4096 < body + scratch
    sums = []
    for budget in (1 << 30, short + 4096):
        p = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, TALSH_B200_GPU_BUDGET_BYTES=str(budget)),
                           stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
        assert p.returncode == 0 and " deferred 0;" in p.stdout, p.stdout
        sums.append([x for x in p.stdout.splitlines() if x.startswith("sum")])
    assert len(sums[0]) == 1 and sums[0] == sums[1]


# 128 x 128 R4 tiles (at least two per SM): K whole, and cut in two; both remainders
@pytest.mark.parametrize("m,n,k", [(2209, 2241, 300), (4665, 957, 4001)])
def test_large_r4_tiles(talsh, m, n, k):
    """The wide R4 tiles against 64 bits for both load directions of both operands, accumulating and overwriting, and
    bit for bit against a batch (64 x 64 tiles)."""
    torch = pytest.importorskip("torch")
    lib = T.lib()
    g = torch.Generator(device="cuda")
    g.manual_seed(17)
    s = torch.cuda.current_stream().cuda_stream
    mk = lambda *x: torch.rand(*x, device="cuda", generator=g).mul_(2.0).sub_(1.0)  # noqa: E731
    for l_along_k, r_along_k, acc in [(0, 0, 1), (1, 1, 0), (0, 1, 0), (1, 0, 1)]:
        # row-major (cols, rows) is the column-major (rows, cols) body
        l, r, d0 = mk(m, k) if l_along_k else mk(k, m), mk(n, k) if r_along_k else mk(k, n), mk(n, m)
        ld, rd = ([k, m] if l_along_k else [m, k]), ([k, n] if r_along_k else [n, k])
        cptrn = ([-(1 if r_along_k else 2), 1] if l_along_k else [1, -(1 if r_along_k else 2)]) + \
            ([-(1 if l_along_k else 2), 2] if r_along_k else [2, -(1 if l_along_k else 2)])
        args = (T.R4, T.ivec(cptrn), 2, T.ivec([m, n]), 2, T.ivec(ld), 2, T.ivec(rd))
        need = lib.tcTensorContractScratch(*args)
        assert (need > (16 * (m + n + k) + 255) // 256 * 256) == (k > 1000)  # cut or whole
        buf = torch.empty(need, dtype=torch.uint8, device="cuda")
        d, d2 = d0.clone(), d0.clone()
        assert lib.tcTensorContract(*args, d.data_ptr(), l.data_ptr(), r.data_ptr(), 0.5, 0.0, 0, acc, buf.data_ptr(),
                                    need, s) == 0
        a, b = (l if l_along_k else l.T).double(), (r if r_along_k else r.T).double()
        ref = 0.5 * (b @ a.T) + (d0.double() if acc else 0.0)
        assert float(torch.linalg.norm(d.double() - ref) / torch.linalg.norm(ref)) <= TOL[T.R4]
        t = (T.ContractTask * 1)()
        t[0].data_kind, t[0].drank, t[0].lrank, t[0].rrank = T.R4, 2, 2, 2
        for to, v in ((t[0].cptrn, cptrn), (t[0].ddims, [m, n]), (t[0].ldims, ld), (t[0].rdims, rd)):
            for i, x in enumerate(v):
                to[i] = x
        t[0].D, t[0].L, t[0].R = d2.data_ptr(), l.data_ptr(), r.data_ptr()
        t[0].alpha_re, t[0].accumulative = 0.5, acc
        need = lib.tcTensorContractBatchScratch(1, t)
        buf = torch.empty(need, dtype=torch.uint8, device="cuda")
        assert lib.tcTensorContractBatch(1, t, buf.data_ptr(), need, s) == 0
        torch.cuda.synchronize()
        assert torch.equal(d, d2)
