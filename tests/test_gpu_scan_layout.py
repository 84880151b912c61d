"""The look-back scan where its rows change form: whole and ragged tiles (8,192
elements), rows of a warp cut anywhere, arrays that are not 16-byte aligned,
more tiles than one look-back window or one wave of CTAs."""
import numpy as np
import pytest

import psb200
from oracle import ps_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 127, 129, 1023, 1025, 8192, 8193, 3 * 8192 - 1, 129 * 8192 + 5, 700 * 8192])
@pytest.mark.parametrize("skip_in,skip_out", [(0, 0), (1, 0), (0, 3), (2, 2)])
def test_scan_of_unaligned_arrays(need_gpu, n, skip_in, skip_out):
    import torch

    rng = np.random.default_rng(n + 10 * skip_in + skip_out)
    a = rng.integers(0, 5, size=n, dtype=np.uint32)
    d_in = torch.zeros(n + 8, dtype=torch.int32, device="cuda")
    d_in[skip_in:skip_in + n] = torch.from_numpy(a.view(np.int32)).cuda()
    d_out = torch.full((n + 8,), -1, dtype=torch.int32, device="cuda")
    scratch = torch.empty(psb200.exclusive_scan_scratch_bytes(n), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    psb200.exclusive_scan_u32(d_in.data_ptr() + 4 * skip_in, d_out.data_ptr() + 4 * skip_out, n, scratch.data_ptr(), 0)
    torch.cuda.synchronize()
    got = d_out.cpu().numpy()
    assert np.array_equal(got[skip_out:skip_out + n].view(np.uint32), O.exclusive_scan(a))
    assert (got[:skip_out] == -1).all() and (got[skip_out + n:] == -1).all()  # nothing beside the array
