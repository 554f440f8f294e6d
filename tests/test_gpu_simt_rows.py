"""The SIMT step at fp32 head_dim 256 with two and with four rows a thread (by the number of blocks), against attention in 64
bits: ragged rows and keys, causal and document masks, segment maps with a stride, a state that goes on."""
import numpy as np
import pytest
import torch

from ring_attention_b200 import api
from ring_attention_b200._lib import SegMap
from util import normal_inputs

pytestmark = pytest.mark.gpu


def positions(bases, seg_len, n, stride):
    return np.array([bases[i // seg_len] + i % seg_len * stride for i in range(n)])


@pytest.mark.parametrize("H,kvH,Sq", [(16, 4, 601), (16, 16, 640), (2, 1, 601), (150, 2, 64), (3, 3, 1)])
@pytest.mark.parametrize("causal,doc,bases,stride,Sk", [
    (False, 0, (0,), 1, 333), (True, 0, (0,), 1, 641), (True, 100, (0,), 1, 601), (True, 0, (0, 400), 1, 640),
    (True, 0, (3,), 4, 607), (False, 0, (0,), 1, 31)])
def test_simt_rows_against_64_bits(H, kvH, Sq, causal, doc, bases, stride, Sk):
    D = 256
    q, k, v = normal_inputs(41, 1, H, kvH, Sq, Sk, D)
    qp, kp = positions((0,), Sq, Sq, stride), positions(bases, Sk // len(bases), Sk, stride)
    seen = np.ones((Sq, Sk), bool) if not causal else kp[None] <= qp[:, None]
    if doc:
        seen &= kp[None] // doc == qp[:, None] // doc
    of = torch.arange(H) % kvH
    q64, k64, v64 = (torch.from_numpy(x.astype(np.float64)) for x in (q, k, v))
    s = (q64 @ k64[:, of].transpose(-1, -2)) / D ** 0.5
    size = ((q64.abs() @ k64[:, of].abs().transpose(-1, -2)) / D ** 0.5).max().item()
    w = torch.softmax(s.masked_fill(~torch.from_numpy(seen), -np.inf), -1).nan_to_num(0.0)
    want = (w @ v64[:, of]).numpy()
    # scores: 16 products a lane, four merges; weights: exponential of 2 ulp; one addition a key on O and l
    eps = 2.0 ** -24
    tol = (2 * (24 * eps * size + 4 * eps) + 2 * (Sk + 16) * eps) * np.abs(v).max()
    dq = torch.from_numpy(q).cuda()
    out = torch.full((1, H, Sq, D), float("nan"), device="cuda")
    m, l = (torch.empty((1, H, Sq), device="cuda") for _ in range(2))
    cut = Sk // 3 // 2 * 2 + 1 if Sk > 32 and len(bases) == 1 else Sk
    for lo, hi in ((0, cut), (cut, Sk)):  # the second part goes on with the state of the first
        if lo == hi:
            continue
        dk, dv = (torch.from_numpy(np.ascontiguousarray(x[:, :, lo:hi])).cuda() for x in (k, v))
        api.attention_step_ex(dq, dk, dv, out, m, l, api.AttentionShape(1, H, Sq, hi - lo, D, kvH), SegMap.make([0], Sq),
                              SegMap.make([b + lo * stride for b in bases], (hi - lo) // len(bases)), pos_stride=stride, causal=causal, fresh=lo == 0,
                              finalize=hi == Sk, doc_len=doc)
    assert np.abs(out.cpu().numpy() - want).max() <= tol
