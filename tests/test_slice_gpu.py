"""Tensor slicing and insertion on the GPU (tcTensorSlice / tcTensorInsert and
talshTensorSlice / talshTensorInsert) against the oracle's restatement of
tensor_block_slice / tensor_block_insert: bit-exact, every kind."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
import tal_sh_b200 as T
from gpu_util import fort, host_tensor, rand

pytestmark = pytest.mark.gpu

KINDS = [T.R4, T.R8, T.C4, T.C8]


def _case(rng, r, long_run=False):
    """Full extents with a volume of at most about 2^20 elements."""
    top = max(2, int(round((1 << 20) ** (1.0 / r))))
    full = [int(rng.integers(1, top + 1)) for _ in range(r)]
    if long_run:
        full[0] = 300
        for i in range(1, r):
            full[i] = min(full[i], max(1, int(((1 << 20) / 300) ** (1.0 / max(r - 1, 1)))))
    sl = [int(rng.integers(1, f + 1)) for f in full]
    if long_run:
        sl[0] = full[0]  # a fully covered leading dimension fuses into the run
    off = [int(rng.integers(0, f - s + 1)) for f, s in zip(full, sl)]
    return full, sl, off


def _dev(torch, a):
    return torch.from_numpy(np.asarray(a).ravel(order="F").copy()).cuda()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("r", [1, 2, 3, 4, 6])
def test_device_slice_insert_bit_exact(talsh, kind, r):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(r * 31 + kind)
    L = T.lib()
    s = torch.cuda.current_stream().cuda_stream
    for long_run in (False, True):
        full, sl, off = _case(rng, r, long_run)
        F, S0 = rand(full, kind, rng), rand(sl, kind, rng)
        for acc in (0, 1):
            # slice
            f, d = _dev(torch, F), _dev(torch, S0)
            assert L.tcTensorSlice(kind, r, T.ivec(full), T.ivec(sl), T.ivec(off), f.data_ptr(), d.data_ptr(),
                                   acc, s) == 0
            want = S0.copy(order="F")
            assert O.tensor_slice(want, F, off, bool(acc)) == 0
            torch.cuda.synchronize()
            assert np.array_equal(d.cpu().numpy().reshape(sl, order="F"), want), (full, sl, off, acc)
            # insert
            f = _dev(torch, F)
            d = _dev(torch, S0)
            assert L.tcTensorInsert(kind, r, T.ivec(full), T.ivec(sl), T.ivec(off), d.data_ptr(), f.data_ptr(),
                                    acc, s) == 0
            want = F.copy(order="F")
            assert O.tensor_insert(want, S0, off, bool(acc)) == 0
            torch.cuda.synchronize()
            assert np.array_equal(f.cpu().numpy().reshape(full, order="F"), want), (full, sl, off, acc)


def test_device_slice_rejects_out_of_range(talsh):
    L = T.lib()
    args = (T.R8, 2, T.ivec([4, 4]), T.ivec([3, 3]))
    assert L.tcTensorSlice(*args, T.ivec([2, 0]), 1, 1, 0, None) == T.TALSH_INVALID_ARGS
    assert L.tcTensorInsert(*args, T.ivec([0, -1]), 1, 1, 0, None) == T.TALSH_INVALID_ARGS


@pytest.mark.parametrize("kind", [T.R8, T.C8])
def test_talsh_slice_and_insert(talsh, kind):
    """talshTensorSlice / talshTensorInsert (talsh.h API, Host tensors staged to GPU 0)."""
    rng = np.random.default_rng(4)
    full, sl, off = [17, 9, 23], [5, 9, 11], [3, 0, 7]
    F, S0 = rand(full, kind, rng), rand(sl, kind, rng)
    Lb = T.lib()
    for acc in (T.NOPE, T.YEP):
        S = S0.copy(order="F")
        dt, lt = host_tensor(S), host_tensor(F)
        assert Lb.talshTensorSlice(dt.ref, lt.ref, T.ivec(off), 0, T.DEV_NVIDIA_GPU, T.COPY_TT, acc, None) == 0
        dt.destruct(); lt.destruct()
        want = S0.copy(order="F")
        assert O.tensor_slice(want, F, off, acc == T.YEP) == 0
        assert np.array_equal(S, want)
        G = F.copy(order="F")
        dt, lt = host_tensor(G), host_tensor(S0)
        assert Lb.talshTensorInsert(dt.ref, lt.ref, T.ivec(off), 0, T.DEV_NVIDIA_GPU, T.COPY_TT, acc, None) == 0
        dt.destruct(); lt.destruct()
        want = F.copy(order="F")
        assert O.tensor_insert(want, S0, off, acc == T.YEP) == 0
        assert np.array_equal(G, want)
    # a slice that does not fit is refused before any work
    S = fort(np.zeros([5, 9, 11], dtype=F.dtype))
    dt, lt = host_tensor(S), host_tensor(F)
    assert Lb.talshTensorSlice(dt.ref, lt.ref, T.ivec([13, 0, 0]), 0, T.DEV_NVIDIA_GPU, T.COPY_TT, T.NOPE,
                               None) == T.TALSH_INVALID_ARGS
    dt.destruct(); lt.destruct()


@pytest.mark.parametrize("kind", KINDS)
def test_slice_insert_units(talsh, kind):
    """Every copy unit (16, 8 bytes, one element): runs, origins, strides or bodies that only the narrower ones
    divide, against numpy, bit-exact; fully covered middle dimensions continue the one before."""
    torch = pytest.importorskip("torch")
    L, rng = T.lib(), np.random.default_rng(77)
    s = torch.cuda.current_stream().cuda_stream
    cases = [([64, 9, 5], [32, 9, 5], [16, 0, 0]), ([64, 9, 5], [32, 4, 5], [2, 1, 0]), ([62, 9, 5], [31, 4, 2], [3, 1, 0]),
             ([12, 7, 6, 4], [8, 7, 6, 2], [4, 0, 0, 1]), ([2051], [1026], [1]), ([5, 1, 7], [4, 1, 7], [0, 0, 0]),
             ([6, 8, 3, 3], [6, 8, 1, 2], [0, 0, 2, 1])]
    for (full, sl, off), shift in [(c, k) for c in cases for k in (0, 1)]:
        F, S = rand(full, kind, rng), rand(sl, kind, rng)
        where = tuple(slice(o, o + n) for o, n in zip(off, sl))
        for insert in (False, True):
            for acc in (0, 1):
                a, b = (S, F) if insert else (F, S)
                ref = b.copy(order="F")
                if insert:
                    ref[where] = ref[where] + a if acc else a
                else:
                    ref[...] = ref + a[where] if acc else a[where]
                bufs = []
                for x in (a, b):
                    t = torch.empty(x.size + shift, dtype=_dev(torch, x).dtype, device="cuda")[shift:]
                    t.copy_(_dev(torch, x))
                    bufs.append(t)
                fn = L.tcTensorInsert if insert else L.tcTensorSlice
                rc = fn(kind, len(full), T.ivec(full), T.ivec(sl), T.ivec(off), bufs[0].data_ptr(), bufs[1].data_ptr(),
                        acc, s)
                torch.cuda.synchronize()
                assert rc == 0 and bufs[1].cpu().numpy().tobytes() == ref.tobytes(order="F"), (full, sl, off, shift,
                                                                                                  insert, acc)


def test_slice_insert_past_32_bits(talsh):
    """More than 2^31 one-element units (64-bit unit numbers): a 2 x 1100000000 R4 slice of a 3 x 1100000001 tensor and
    its insertion, bit-exact."""
    torch = pytest.importorskip("torch")
    L, n = T.lib(), 1100000000
    s = torch.cuda.current_stream().cuda_stream
    full = torch.empty(3 * (n + 1), dtype=torch.int32, device="cuda")
    step = 1 << 27
    pieces = range(0, n, step)  # filled and compared in pieces: the temporaries stay small
    for lo in range(0, full.numel(), step):
        hi = min(lo + step, full.numel())
        full[lo:hi] = torch.arange(lo, hi, device="cuda") % 2000000011
    part = torch.zeros(2 * n, dtype=torch.int32, device="cuda")
    args = (T.R4, 2, T.ivec([3, n + 1]), T.ivec([2, n]), T.ivec([1, 0]))
    assert L.tcTensorSlice(*args, full.data_ptr(), part.data_ptr(), 0, s) == 0
    want = full.view(n + 1, 3)[:n, 1:]
    got = part.view(n, 2)
    assert all(torch.equal(got[lo:lo + step], want[lo:lo + step]) for lo in pieces)
    # few units at offsets past 2^31
    few = torch.zeros(2 * 1000, dtype=torch.int32, device="cuda")
    assert L.tcTensorSlice(T.R4, 2, T.ivec([3, n + 1]), T.ivec([2, 1000]), T.ivec([1, n - 999]), full.data_ptr(),
                           few.data_ptr(), 0, s) == 0
    assert torch.equal(few.view(1000, 2), full.view(n + 1, 3)[n - 999:, 1:])
    part.bitwise_not_()
    assert L.tcTensorInsert(*args, part.data_ptr(), full.data_ptr(), 0, s) == 0
    rows = full.view(n + 1, 3)
    for lo in pieces:
        hi = min(lo + step, n)
        assert torch.equal(rows[lo:hi, 1:], got[lo:hi])
        assert torch.equal(rows[lo:hi, 0].long(), torch.arange(3 * lo, 3 * hi, 3, device="cuda") % 2000000011)
