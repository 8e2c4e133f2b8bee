"""BF16 shadows at the edges of the conversion routine: the source's last rows and columns inside and at
the end of an 8-column word, sources narrower than a word, strides and offsets that allow 32-byte loads
or not, every chunk height, plain and split; values at ties, in FP32's and BF16's subnormal range and
near overflow.  The bytes are the oracle's."""
import numpy as np
import pytest
import torch

from test_gpu_bf16 import SPLIT_A, SPLIT_B, dev, ptr, shadow_task

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [0, SPLIT_A, SPLIT_B])
@pytest.mark.parametrize("cr,rows", [(32, 32), (64, 128), (128, 256)])
@pytest.mark.parametrize("transposed,mr,nc,pad,off", [(0, 0, 0, 0, 0), (0, 31, 60, 0, 0), (0, 1, 7, 1, 0), (0, 17, 57, 4, 4),
                                                      (0, 32, 64, 2, 0), (0, 30, 9, 4, 2), (1, 0, 0, 0, 0), (1, 31, 57, 1, 3)])
def test_edges(pp, oracle, gctx, transposed, mr, nc, pad, off, cr, rows, split):
    rng = np.random.default_rng(rows + mr + nc)
    K, r, c = 128, mr or rows, nc or 128
    x = rng.standard_normal((c, r + pad) if transposed else (r, c + pad))
    x *= 10.0 ** rng.integers(-42, 37, x.shape)
    ties = rng.integers(0, 4, x.shape) == 0
    x[ties] = (1 + (2 * rng.integers(0, 128, x.shape) + 1) * 2.0**-8)[ties]
    x[rng.integers(0, 9, x.shape) == 0] = -0.0
    src = np.concatenate([np.zeros(off), x.ravel()])
    out = []
    for side in ("dev", "host"):
        words = rows * K * (3 if split else 1) // 4
        sh = torch.full((words,), 7.0, dtype=torch.float64, device="cuda") if side == "dev" else np.full(words, 7.0)
        s = dev(src) if side == "dev" else src
        t = shadow_task(pp, ptr(sh), ptr(s) + 8 * off, rows, K * (3 if split else 1), transposed, x.shape[1])
        t[0]["l"], t[0]["n"], t[0]["o"], t[0]["ctrl"] = mr, nc, split, 0 if cr == 128 else cr
        if side == "dev":
            gctx.vm_execute(t, np.zeros(0, np.int32), np.zeros(1, np.int32))
            out.append(sh.cpu().numpy())
        else:
            assert oracle.lib().oracle_run_program(t.ctypes.data, 1) == 0
            out.append(sh)
    assert np.array_equal(out[0].view(np.uint16), out[1].view(np.uint16))
