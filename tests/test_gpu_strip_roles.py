"""The roles of the strip kernels at the ends of what they hand each other: streams of blocks shorter and longer than the
batch the masking warp works out, the record rings and the rings of keys and values."""
import pytest
from test_gpu_strips import test_strips_against_simt as against_simt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("th,tw,b,wr,wc,dqk,dv,R,BH", [
    (1, 8, 1, 0, 0, 64, 64, 0, 1), (2, 8, 1, 1, 1, 64, 64, 16, 1), (5, 9, 1, 1, 1, 64, 64, 16, 149), (32, 8, 1, 0, 1, 64, 64, 8, 1),
    (33, 8, 1, 3, 3, 64, 64, 16, 2), (257, 8, 1, 2, 2, 64, 64, 16, 1), (4, 8, 1, 1, 1, 128, 128, 32, 1), (17, 24, 1, 9, 15, 128, 128, 32, 3),
    (70, 20, 1, 12, 12, 128, 128, 16, 60), (19, 31, 1, 7, 7, 128, 64, 16, 9), (40, 17, 1, 15, 15, 96, 96, 8, 40), (8, 8, 16, 1, 1, 32, 32, 0, 2)])
def test_streams_of_any_length(th, tw, b, wr, wc, dqk, dv, R, BH):
    against_simt(th, tw, b, wr, wc, dqk, dv, R, BH)
