"""Ranking of a beam-search step on both sides of the largest cluster (16 hypotheses), against the torch implementation."""

import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("beam", [1, 2, 3, 9, 15, 16, 17])
@pytest.mark.parametrize("k,V,kind", [(1, 7, "plain"), (16, 3, "plain"), (12, 5121, "plain"), (8, 4000, "equal"), (32, 1000, "finished"), (5, 33, "lowest"), (4, 160000, "plain")])
def test_beam_topk_cluster(beam, k, V, kind):
    from returnn_b200.ops import seq_ops

    torch.manual_seed(beam * 100 + k)
    B = 4
    logits = torch.randn(B, beam, V, device="cuda") * 3
    prev = -torch.rand(B, beam, device="cuda") * 5
    fin = torch.rand(B, beam, device="cuda") < 0.2
    if kind == "equal":
        logits[:] = 1.0  # more equal values than the list of candidates holds
    if kind == "finished":
        fin[:] = True
    if kind == "lowest":
        logits[:, :, ::2] = torch.finfo(torch.float32).min
    s, back, lab = seq_ops.beam_topk(logits, prev, finished=fin, eos=2, k=k)
    n = min(k, int((~fin).sum(1).min()) * V + int(fin.sum(1).min()))  # continuations that every entry has
    rs, rback, rlab = seq_ops.beam_topk_reference(logits, prev, fin, 2, min(k, beam * V))
    torch.testing.assert_close(s[:, :n], rs[:, :n], atol=2e-3, rtol=1e-4)
    # the score of what is named is the score that is given (ties may be resolved otherwise by the reference)
    logp = torch.log_softmax(logits, -1) + prev[:, :, None]
    named = logp[torch.arange(B, device="cuda")[:, None], back[:, :n].long(), lab[:, :n].long()]
    named = torch.where(fin.gather(1, back[:, :n].long()), prev.gather(1, back[:, :n].long()), named)
    torch.testing.assert_close(named, s[:, :n], atol=2e-3, rtol=1e-4)
    key = (back.long() * V + lab.long())[:, :n]
    assert all(len(set(row.tolist())) == n for row in key)
