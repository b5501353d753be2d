"""Contractions whose free indices are walked in D's order (the operand's stride-1 index is contracted, or K is
short and D's fastest index does not lead its group, where that moves fewer sectors): against numpy in 64 bits on both
sides of the rule, alone and bit for bit in a batch."""
import re

import numpy as np
import pytest

import tal_sh_b200 as T
from gpu_util import rand, rel_err

pytestmark = pytest.mark.gpu

TOL = {T.R8: 1e-12, T.C8: 1e-12, T.R4: 2e-5, T.C4: 2e-5}  # the parity bars of every contraction test
CASES = [("D(a,b,c,d)+=L(e,b,a,d)*R(c,e)", dict(a=13, b=9, c=11, d=7, e=17)),
         ("D(a,b,c,d)+=L(e,b,a,d)*R(c,e)", dict(a=5, b=17, c=3, d=9, e=131)),
         ("D(a,b,c,d,e,f)+=L(d,e,g,a)*R(g,f,b,c)", dict(a=7, b=5, c=6, d=9, e=3, f=4, g=19)),
         ("D(a,b,c,d,e,f)+=L(d,e,g,a)*R(g,f,b,c)", dict(a=9, b=3, c=5, d=7, e=2, f=6, g=383)),
         ("D(a,b,c,d,e,f)+=L(d,e,g,a)*R(g,f,b,c)", dict(a=9, b=3, c=5, d=7, e=2, f=6, g=384)),
         ("D(b,a,d,c)+=L(c,k,d)*R(a,k,b)", dict(a=21, b=13, c=11, d=9, k=15)),
         ("D(b,a,h,d,c)+=L(c,k,h,d)*R(a,k,h,b)", dict(a=11, b=13, c=8, d=9, k=15, h=3)),
         # outputs thin one way, where the line moves with the width: operand's order and D's
         ("D(e,m)+=L(m,k,e,c)*R(c,k)", dict(m=17, k=15, e=70, c=20)),
         ("D(e,m,i)+=L(m,k,e,c)*R(c,k,i)", dict(m=17, k=2, e=70, c=3, i=8)),
         ("D(e,m,i)+=L(m,k,e,c)*R(c,k,i)", dict(m=17, k=15, e=70, c=20, i=8)),
         ("D(e,m,i)+=L(m,k,e,c)*R(c,k,i)", dict(m=17, k=4, e=70, c=5, i=65)),
         ("D(e,m,i)+=L(k,m,e,c)*R(c,k,i)", dict(m=17, k=2, e=70, c=100, i=3)),
         ("D(j,i,a)+=L(k,a)*R(i,j,k)", dict(i=70, j=33, k=40, a=2))]


@pytest.mark.parametrize("kind", [T.R4, T.R8, T.C4, T.C8])
def test_free_index_order(talsh, kind):
    torch = pytest.importorskip("torch")
    lib, rng = T.lib(), np.random.default_rng(13)
    s = torch.cuda.current_stream().cuda_stream
    dev = lambda a: torch.from_numpy(np.asarray(a).ravel(order="F").copy()).cuda()
    tasks, keep = (T.ContractTask * len(CASES))(), []
    for t, (pattern, ext) in zip(tasks, CASES):
        di, li, ri = ([x for x in g.split(",")] for g in re.findall(r"\(([a-z,]*)\)", pattern))
        dd, ld, rd = ([ext[x] for x in g] for g in (di, li, ri))
        D0, L, R = (rand(x, kind, rng) for x in (dd, ld, rd))
        e, dig, dr, lr, rr, _ = T.parse_pattern(pattern)
        assert e == 0
        d, d2, l, r = dev(D0), dev(D0), dev(L), dev(R)
        args = (kind, T.ivec(dig), dr, T.ivec(dd), lr, T.ivec(ld), rr, T.ivec(rd))
        need = lib.tcTensorContractScratch(*args)
        buf = torch.empty(need, dtype=torch.uint8, device="cuda")
        assert lib.tcTensorContract(*args, d.data_ptr(), l.data_ptr(), r.data_ptr(), 0.5, 0.0, 0, 1, buf.data_ptr(),
                                    need, s) == 0
        torch.cuda.synchronize()
        wide = np.complex128
        ref = D0.astype(wide) + 0.5 * np.einsum("%s,%s->%s" % ("".join(li), "".join(ri), "".join(di)), L.astype(wide),
                                                R.astype(wide))
        assert rel_err(d.cpu().numpy().reshape(dd, order="F"), ref) <= TOL[kind], (pattern, ext)
        t.data_kind, t.drank, t.lrank, t.rrank = kind, dr, lr, rr
        for to, xs in ((t.cptrn, dig), (t.ddims, dd), (t.ldims, ld), (t.rdims, rd)):
            for i, v in enumerate(xs):
                to[i] = v
        t.D, t.L, t.R = d2.data_ptr(), l.data_ptr(), r.data_ptr()
        t.alpha_re, t.alpha_im, t.conj_bits, t.accumulative = 0.5, 0.0, 0, 1
        keep.append((d, d2, l, r))
    need = lib.tcTensorContractBatchScratch(len(CASES), tasks)
    buf = torch.empty(need, dtype=torch.uint8, device="cuda")
    assert lib.tcTensorContractBatch(len(CASES), tasks, buf.data_ptr(), need, s) == 0
    torch.cuda.synchronize()
    for (d, d2, _, _), case in zip(keep, CASES):
        assert torch.equal(d, d2), case
