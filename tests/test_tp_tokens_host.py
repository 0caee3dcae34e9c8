"""The rule by which the tensor-parallel GPU test compares the tokens of two runs."""
import torch

from _tp_worker import LOGIT_BOUND, same_tokens


def test_tokens_may_part_only_at_a_near_tie():
    a = torch.tensor([[3, 1, 4, 1], [5, 9, 2, 6]])
    asked = []

    def behind(gap):
        def logits(s, tokens):
            asked.append((s, tokens.tolist()))
            lg = torch.zeros(10)
            lg[4], lg[7] = 1.0, 1.0 - gap
            return lg
        return logits

    assert same_tokens(a, a.clone(), behind(1.0)) and asked == []
    b = a.clone()
    b[0, 2:] = torch.tensor([7, 8])                     # parts at the third token; what follows is another context
    assert same_tokens(a, b, behind(1.9 * LOGIT_BOUND)) and asked == [(0, [3, 1])]
    assert same_tokens(a, b, behind(-1.9 * LOGIT_BOUND))
    assert not same_tokens(a, b, behind(2.1 * LOGIT_BOUND))
