"""The roles of the strip kernels at the ends of what they hand each other: streams of blocks shorter and longer than the
batch the masking warp works out, the record rings and the rings of keys and values; rows whose maximum lies outside the
columns that the forward kernel starts from."""
import pytest
import torch

from oracle import swa_oracle as orc
from test_gpu_strips import test_strips_against_simt as against_simt

import dl_templates_b200 as swa

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("th,tw,b,wr,wc,dqk,dv,R,BH", [
    (1, 8, 1, 0, 0, 64, 64, 0, 1), (2, 8, 1, 1, 1, 64, 64, 16, 1), (5, 9, 1, 1, 1, 64, 64, 16, 149), (32, 8, 1, 0, 1, 64, 64, 8, 1),
    (33, 8, 1, 3, 3, 64, 64, 16, 2), (257, 8, 1, 2, 2, 64, 64, 16, 1), (4, 8, 1, 1, 1, 128, 128, 32, 1), (17, 24, 1, 9, 15, 128, 128, 32, 3),
    (70, 20, 1, 12, 12, 128, 128, 16, 60), (19, 31, 1, 7, 7, 128, 64, 16, 9), (40, 17, 1, 15, 15, 96, 96, 8, 40), (8, 8, 16, 1, 1, 32, 32, 0, 2)])
def test_streams_of_any_length(th, tw, b, wr, wc, dqk, dv, R, BH):
    against_simt(th, tw, b, wr, wc, dqk, dv, R, BH)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("th,tw,wr,wc", [(24, 24, 6, 6), (19, 35, 6, 5), (40, 9, 5, 6)])
@pytest.mark.parametrize("big", [8., 40.])
def test_maxima_outside_the_first_columns_looked_at(th, tw, wr, wc, big, dtype):
    """Keys of every other grid row (and column) are large, the others small: the running maximum that a row starts from is far
    below its true one -- by more than any 16-bit type holds, with the larger factor -- and has to be replaced.  The result is
    close to single rows of v: |v| < 4.5, so P and the output, rounded to 8 (11) bits, are off by 2^-9 (2^-12) of it each."""
    q, k, v, do = orc.seeded_inputs(1, 2, th * tw, 64, 64, dtype, th + tw)
    n = torch.arange(th * tw)
    for sel in ((n // tw) % 2 == 0, (n % tw) % 3 == 0, n % tw < tw - 4):
        ks = torch.where(sel[:, None], k.float() * big, k.float() * 0.05).to(dtype)
        want = orc.fused_ref(q.float(), ks.float(), v.float(), do.float(), None, None, None, 1, th, tw, wr, wc, 0.125)[0]
        o, lse = swa.swa_forward(q.to(DEV), ks.to(DEV), v.to(DEV), None, 1, th, tw, wr, wc, 0.125, impl="tc")
        swa.check_status()
        assert torch.isfinite(lse).all()
        assert orc.max_abs(o.float().cpu(), want) < 2e-2
