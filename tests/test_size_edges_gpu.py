"""Every kernel variant that a size rule selects, at the sizes where it can go wrong: edges of its tiles, remainders, the
smallest and largest of its range and the first size of the next variant."""
import numpy as np
import pytest
import torch

import void_b200 as void
from oracle import void_oracle as vo

pytestmark = pytest.mark.gpu


# ------------------------------------------------------------------------------------------ columns quantised
@pytest.mark.parametrize("k,n", [(1, 1), (7, 5), (8, 16), (33, 17), (513, 36), (8192, 12), (8193, 288), (8200, 292),
                                 (26624, 40), (26632, 40), (30000, 3)])
def test_quantised_columns_match_the_oracle_bits(k, n):
    gen = torch.Generator().manual_seed(k * 1000 + n)
    b = torch.randn(k, n, generator=gen)
    b[:, 0] = torch.randint(-256, 257, (k,), generator=gen) * 0.5         # scale 1: quotients on half integers ...
    b[0, 0] = 128.0
    if k > 8:
        b[5, 0] = float(np.nextafter(np.float32(2.5), np.float32(3)))
        b[6, 0] = float(np.nextafter(np.float32(-3.5), np.float32(0)))
    b[:, n // 2] *= 0 if n > 1 else 1                                     # ... and a column of zeros
    q, s = void.quantize_cols_int8(b.cuda())
    ref_q, ref_s = vo.quantize_int8_cols(b.numpy())
    assert np.array_equal(s.cpu().numpy(), ref_s) and np.array_equal(q.cpu().numpy(), ref_q)
    f, fs, fi = void.quantize_cols_fp8(b.cuda())
    ref_f, ref_fs, ref_fi = vo.quantize_fp8_cols(b.numpy())
    assert np.array_equal(fs.cpu().numpy(), ref_fs) and np.array_equal(fi.cpu().numpy(), ref_fi)
    assert np.array_equal(f.view(torch.uint8).cpu().numpy(), ref_f)
    off = torch.zeros(k, n + 3).cuda()[:, 1:n + 1]                        # rows that start off 16-byte boundaries
    off.copy_(b)
    assert torch.equal(void.quantize_cols_int8(off)[0], q)
