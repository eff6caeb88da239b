"""Recorded passes (ops/graph.py) give what the launches one by one give, over changing inputs, carries and step scalars."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu

from gruboros_b200.optim.schedulefree import AdamWScheduleFree
from gruboros_b200.runtime.trainer import Trainer
from tests.test_engine_gpu import make_pair
from tests.test_model_cpu import zipf_bytes


@pytest.mark.parametrize("B,chunk,accum", [(1, 3, 1), (2, 65, 1), (3, 130, 2)])
def test_recorded_training_equals_single_launches(B, chunk, accum):
    a, _ = make_pair(dim=128, depth=3)
    b = copy.deepcopy(a)
    b.fused_engine()._recordable = lambda: False
    trainers = []
    for m in (a, b):
        opt = AdamWScheduleFree(m.parameters(), lr=1e-3, betas=(0.9, 0.995), weight_decay=1e-4, warmup_steps=4)
        opt.train()
        trainers.append(Trainer(m, opt, chunk_size=chunk, grad_accum=accum))
    losses = [[], []]
    for r in range(3):                                   # 12 chunks, the carry dropped between sequences
        x = zipf_bytes(B, 4 * chunk, seed=r).cuda()
        for t, l in zip(trainers, losses):
            l += t.train_sequence(x)
    la, lb = torch.stack(losses[0]), torch.stack(losses[1])
    # atomics add gradients in any order (fp32 rounding, 2^-24 of each term); Adam's normalised step of the first updates
    # turns a gradient's relative error into the same relative error of a step of size lr
    assert (la - lb).abs().max().item() < 2e-3
    d = (a.fused_engine().flat.data - b.fused_engine().flat.data).abs()
    assert d.max().item() < 1e-2 and d.mean().item() < 2e-5
    ka, kb = (t.optimizer.param_groups[0]["k"] for t in trainers)
    assert ka == kb == 12 // accum
    assert any(v for bufs in a.fused_engine()._bufs.values() for v in bufs.recorder._seen.values() if not isinstance(v, int))


def test_recorded_forward_reads_new_tokens_and_weights():
    m, _ = make_pair(dim=128, depth=2)
    with torch.no_grad():
        for r in range(5):
            x = zipf_bytes(2, 33, seed=r).cuda()
            if r == 3:
                m.to_logits.weight.mul_(0.5)
            logits, hid = m(x.long(), return_prev_hiddens=True)
            fresh = copy.deepcopy(m)
            want, hid_w = fresh(x, return_prev_hiddens=True)
            assert torch.equal(logits, want) and all(torch.equal(p, q) for p, q in zip(hid, hid_w))
            _, hid2 = m(x, return_prev_hiddens=True, prev_hiddens=hid)          # consecutive views as the carry
            _, hid3 = fresh(x, return_prev_hiddens=True, prev_hiddens=[h.clone() for h in hid])
            assert all(torch.equal(p, q) for p, q in zip(hid2, hid3))
