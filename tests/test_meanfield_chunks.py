"""GPU: the mean-field kernel at the numbers of 256-column chunks that test_meanfield_sizes.py leaves out (5 and 10), against
the FP64 recurrence with that file's contracting schedule and its bounds."""
import math

import pytest
import torch

from anechoic_b200 import instances as I
from tests.test_meanfield import _case, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,S", [(1025, 18), (1280, 17), (2305, 16), (2560, 33)])
def test_chunks_vs_fp64(cuda, n, S):
    inst = I.random_kbit(n, 2, 900 + n, pzero=0.4, bmax=3)
    theta = (4.0 * math.sqrt(n), math.log(2.0), 1.0, 0.5, 1.05)
    mr = torch.rand(64, n, generator=torch.Generator().manual_seed(3)) * 2 - 1
    r = _case(inst, S, 64, "counted", theta, m0=mr)
    assert (r["mS"] - r["m64"]).abs().max().item() <= 1e-5
    assert _rel(r["g"], r["g64"]) <= 1e-3, (r["g"].tolist(), r["g64"].tolist())
