"""Full contractions (rank-0 D) on the GPU: every index order of R, odd and unit extents, unaligned bodies, conjugation
flags, overwrite and accumulation, against numpy in 64 bits; reruns are bit-identical."""
import itertools

import numpy as np
import pytest

import tal_sh_b200 as T
from gpu_util import rand

pytestmark = pytest.mark.gpu

# the factors are exact in double; |error| <= K eps sum |l r| for any summation order, and one rounding to the kind
EPS = {T.R4: 2.0 ** -24, T.C4: 2.0 ** -24, T.R8: 2.0 ** -53, T.C8: 2.0 ** -53}


def _run(lib, torch, kind, dims, perm, conj, acc, offset=0, rng=None):
    """D (+)= 0.75 * sum L[i] R[perm(i)]; R's dimension j is L's dimension perm[j]."""
    L = rand(dims, kind, rng)
    R = rand([dims[p] for p in perm], kind, rng)
    D0 = rand([1], kind, rng)
    dt = torch.from_numpy(np.zeros(1, T.NP_DTYPE[kind])).dtype

    def dev(a):  # body starting `offset` elements into an allocation
        b = torch.empty(a.size + offset, dtype=dt, device="cuda")[offset:]
        b.copy_(torch.from_numpy(np.asarray(a).ravel(order="F").copy()))
        return b

    l, r = dev(L), dev(R)
    n = len(dims)
    cptrn = [0] * (2 * n)
    for j, p in enumerate(perm):
        cptrn[n + j], cptrn[p] = -(p + 1), -(j + 1)
    args = (kind, T.ivec(cptrn), 0, None, n, T.ivec(dims), n, T.ivec(list(R.shape)))
    need = lib.tcTensorContractScratch(*args)
    buf = torch.empty(need, dtype=torch.uint8, device="cuda")
    outs = []
    for _ in range(2):
        d = torch.from_numpy(D0.copy()).cuda()
        assert lib.tcTensorContract(*args, d.data_ptr(), l.data_ptr(), r.data_ptr(), 0.75, 0.0, conj, acc,
                                    buf.data_ptr(), need, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        outs.append(d.cpu().numpy()[0])
    wide = lambda a: a.astype(np.complex128)
    x, y = wide(L), np.transpose(wide(R), np.argsort(perm))
    x = np.conj(x) if conj & 2 else x
    y = np.conj(y) if conj & 4 else y
    ref = 0.75 * np.sum(x * y) + (complex(D0[0]) if acc else 0.0)
    size = 0.75 * np.sum(np.abs(x) * np.abs(y)) + abs(ref)
    tol = 2 * L.size * EPS[T.R8] * size + 2 * EPS[kind] * (abs(ref) + abs(D0[0]))
    assert outs[0].tobytes() == outs[1].tobytes()
    assert abs(complex(outs[0]) - ref) <= tol, (dims, perm, conj, acc, offset, outs[0], ref)


@pytest.mark.parametrize("kind", [T.R4, T.R8, T.C4, T.C8])
def test_full_contraction(talsh, kind):
    torch = pytest.importorskip("torch")
    lib, rng = T.lib(), np.random.default_rng(8)
    run = lambda *a, **k: _run(lib, torch, kind, *a, rng=rng, **k)
    for perm in itertools.permutations(range(4)):
        run([13, 6, 9, 7], perm, 0, 1)
    for dims, perm in (([1], [0]), ([4], [0]), ([100003], [0]), ([1, 1, 5], [2, 0, 1]), ([513, 511], [1, 0]),
                       ([64, 2, 3, 130], [3, 1, 0, 2]), ([3, 5, 2, 7, 4, 11], [5, 3, 1, 0, 2, 4])):
        for conj in (0, 2, 4, 6):
            run(dims, perm, conj if kind in (T.C4, T.C8) else 0, conj // 2 % 2)
        if kind != T.C8:  # bodies aligned to the element only
            run(dims, perm, 0, 1, offset=1)


def test_long_sums_are_summed_in_parts(talsh):
    """Rounding of 41 M products, 8 draws.  A thread adds about 270 of them: in one chain the error is about
    0.6 u sqrt(n v 270 / 2), v = 1/9 the products' variance (2.6e-16 sqrt(n)); as sums of 8 and then of those, about
    1e-16 sqrt(n).  The line lies at their geometric mean."""
    torch = pytest.importorskip("torch")
    lib = T.lib()
    dims = [80, 64, 100, 80]  # D += L(a,b,i,j) R(b,a,i,j)
    n = int(np.prod(dims))
    args = (T.R8, T.ivec([-2, -1, -3, -4, -2, -1, -3, -4]), 0, None, 4, T.ivec(dims), 4, T.ivec([64, 80, 100, 80]))
    need = lib.tcTensorContractScratch(*args)
    buf = torch.empty(need, dtype=torch.uint8, device="cuda")
    square = 0.0
    for seed in range(8):
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        l, r = (torch.rand(n, dtype=torch.float64, device="cuda", generator=g).mul_(2.0).sub_(1.0) for _ in range(2))
        d = torch.zeros(1, dtype=torch.float64, device="cuda")
        assert lib.tcTensorContract(*args, d.data_ptr(), l.data_ptr(), r.data_ptr(), 1.0, 0.0, 0, 0, buf.data_ptr(),
                                    need, torch.cuda.current_stream().cuda_stream) == 0
        x = l.view(80, 100, 64, 80).cpu().numpy().astype(np.longdouble)
        x *= r.view(80, 100, 80, 64).transpose(2, 3).cpu().numpy()
        square += float((d.cpu().numpy()[0] - x.sum()) ** 2) / n / 8
    assert np.sqrt(square) <= 1.6e-16, np.sqrt(square)
