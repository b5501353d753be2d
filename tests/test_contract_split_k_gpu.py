"""Contractions whose contracted range is split over CTAs (few output tiles, long K): against numpy in 64 bits at
the edges of the split and of the tiles, equal bit for bit alone, repeated and in a batch, and run unsplit when the
scratch has no room for the partial sums."""
import ctypes as C

import numpy as np
import pytest

import tal_sh_b200 as T
from gpu_util import fort, rand, rel_err

pytestmark = pytest.mark.gpu

TOL = {T.R8: 1e-12, T.C8: 1e-12, T.R4: 2e-5, T.C4: 2e-5}  # the parity bars of every contraction test
# (M, N, K): one tile and a remainder each way, K below / at / above two chunks, two-level sums, vectors
SHAPES = [(1, 1, 511), (1, 1, 513), (7, 9, 512), (32, 33, 1023), (40, 40, 20001), (64, 64, 769), (65, 1, 4097),
          (1, 130, 5000), (100, 70, 3000), (200, 150, 1600)]


def _launch(lib, torch, kind, dims, d, l, r, acc, conj=0, scratch=None):
    m, n, k = dims
    args = (kind, T.ivec([-2, 1, 2, -1]), 2, T.ivec([m, n]), 2, T.ivec([k, m]), 2, T.ivec([n, k]))
    need = lib.tcTensorContractScratch(*args)
    size = need if scratch is None else scratch(need, m, n, k)
    buf = torch.empty(size, dtype=torch.uint8, device="cuda")
    rc = lib.tcTensorContract(*args, d.data_ptr(), l.data_ptr(), r.data_ptr(), 0.5, 0.0, conj, acc, buf.data_ptr(),
                              size, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return rc


@pytest.mark.parametrize("kind", [T.R8, T.C8, T.R4, T.C4])
def test_split_k_matches_numpy_alone_and_batched(talsh, kind):
    torch = pytest.importorskip("torch")
    lib, rng = T.lib(), np.random.default_rng(5)
    dev = lambda a: torch.from_numpy(np.asarray(a).ravel(order="F").copy()).cuda()
    tasks = (T.ContractTask * len(SHAPES))()
    keep = []
    for t, (m, n, k) in zip(tasks, SHAPES):
        L, R, D0 = rand([k, m], kind, rng), rand([n, k], kind, rng), rand([m, n], kind, rng)
        conj = 0 if kind in (T.R4, T.R8) else 2  # conj(L)
        ref = D0.astype(np.complex128) + 0.5 * (np.conj(L.astype(np.complex128)).T @ R.astype(np.complex128).T)
        l, r, out = dev(L), dev(R), [dev(D0) for _ in range(4)]
        for d in out[:2]:
            assert _launch(lib, torch, kind, (m, n, k), d, l, r, 1, conj) == 0
        least = lambda need, m, n, k: (16 * (m + n + k) + 255) // 256 * 256  # the offset tables alone
        assert _launch(lib, torch, kind, (m, n, k), out[2], l, r, 1, conj, least) == 0
        short = lambda need, m, n, k: least(need, m, n, k) - 256
        assert _launch(lib, torch, kind, (m, n, k), out[3], l, r, 1, conj, short) == T.TALSH_INVALID_ARGS
        assert torch.equal(out[0], out[1])
        for d in (out[0], out[2]):
            assert rel_err(d.cpu().numpy().reshape(ref.shape, order="F"), ref) <= TOL[kind], (m, n, k)
        t.data_kind, t.drank, t.lrank, t.rrank = kind, 2, 2, 2
        for i, v in enumerate([-2, 1, 2, -1]):
            t.cptrn[i] = v
        for to, dims in ((t.ddims, [m, n]), (t.ldims, [k, m]), (t.rdims, [n, k])):
            for i, v in enumerate(dims):
                to[i] = v
        t.D, t.L, t.R = out[3].data_ptr(), l.data_ptr(), r.data_ptr()
        t.alpha_re, t.alpha_im, t.conj_bits, t.accumulative = 0.5, 0.0, conj, 1
        keep.append((out, l, r))
    need = lib.tcTensorContractBatchScratch(len(SHAPES), tasks)
    buf = torch.empty(need, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    assert lib.tcTensorContractBatch(len(SHAPES), tasks, buf.data_ptr(), need, s) == 0
    torch.cuda.synchronize()
    for (out, _, _), dims in zip(keep, SHAPES):
        assert torch.equal(out[3], out[0]), dims


def test_split_k_with_hyper_indices(talsh):
    """Hyper combinations times splits: D(a,h,b) = L(k,h,a) R(b,k,h), and a recorded batch replayed."""
    torch = pytest.importorskip("torch")
    lib, rng = T.lib(), np.random.default_rng(6)
    a, b, h, k = 33, 18, 5, 3001
    L, R = rand([k, h, a], T.R8, rng), rand([b, k, h], T.R8, rng)
    ref = np.einsum("kha,bkh->ahb", L, R)
    dev = lambda x: torch.from_numpy(np.asarray(x).ravel(order="F").copy()).cuda()
    d, l, r = dev(np.zeros((a, h, b))), dev(L), dev(R)
    args = (T.R8, T.ivec([-2, 2, 1, 3, -1, 2]), 3, T.ivec([a, h, b]), 3, T.ivec([k, h, a]), 3, T.ivec([b, k, h]))
    need = lib.tcTensorContractScratch(*args)
    buf = torch.empty(need, dtype=torch.uint8, device="cuda")
    assert lib.tcTensorContract(*args, d.data_ptr(), l.data_ptr(), r.data_ptr(), 1.0, 0.0, 0, 0, buf.data_ptr(), need,
                                torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert rel_err(d.cpu().numpy().reshape(ref.shape, order="F"), ref) <= TOL[T.R8]
