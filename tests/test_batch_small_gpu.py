"""FP64 batches of small instances: many of them share the queue's two passes
instead of a chain of launches each (csrc/gpp_batch.cu, exact_choice); a few,
and large ones beside them, keep their contractions.  Every output against
the oracle, 1e-12 of its largest value."""
import numpy as np
import pytest

import workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TINY, SMALL, LARGE = (5, 1, 256, 12), (24, 2, 1024, 40), (60, 2, 2048, 60)


@pytest.mark.parametrize("shapes, most", [
    # two reductions; the queue's two passes; eight launches per contraction
    ([SMALL], 12), ([SMALL] * 2, 20), ([SMALL] * 8, 4), ([TINY] * 3, 4), ([LARGE] * 2, 20),
    ([SMALL] * 8 + [LARGE], 12), ([SMALL, TINY, LARGE], 12), ([SMALL, LARGE], 20),
], ids=["1small", "2small", "8small", "3tiny", "2large", "8small1large", "mixed", "1small1large"])
def test_batch_of_small_instances(sigma_lib, shapes, most):
    import torch
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.float64).copy()).cuda()
    probs = [W.gpp_random(nb, nvb, nc, ng, 60 + i) for i, (nb, nvb, nc, ng) in enumerate(shapes)]
    outs, inst = [], []
    for p in probs:
        o = [torch.zeros(n, dtype=torch.float64, device="cuda") for n in (6, 6, 2 * p.number_bands)]
        outs.append(o)
        inst.append(dict(number_bands=p.number_bands, nvband=p.nvband, ncouls=p.ncouls, ngpown=p.ngpown,
                         inv_igp_index=p.inv_igp_index, indinv=p.indinv, wx_array=dev(p.wx_array),
                         aqsmtemp=dev(p.aqsmtemp), aqsntemp=dev(p.aqsntemp), I_eps_array=dev(p.I_eps_array),
                         wtilde_array=dev(p.wtilde_array), vcoul=dev(p.vcoul), achtemp=o[0], asxtemp=o[1],
                         acht_n1_loc=o[2]))
    b = sigma_lib.GppBatch(inst, sigma_lib.PREC_FP64)
    assert b.info()[2] <= most
    b.execute()
    torch.cuda.synchronize()
    assert b.status() == 0
    b.close()
    for p, o in zip(probs, outs):
        for x, y in zip([t.cpu().numpy().view(np.complex128) for t in o], O.gpp(p)):
            assert np.abs(x - y).max() <= 1e-12 * np.abs(y).max()
