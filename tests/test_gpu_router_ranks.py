"""The router's choice among up to 32 experts, which is ranked in registers, by its rules: the largest first, the lowest index among equals,
no number that is none, only the best groups' experts."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rules(z, corr, top, groups, keep, score, rule):
    s = torch.sigmoid(z) if score == "sigmoid" else torch.softmax(z, -1) if score == "softmax" else z
    c = [float(a) + float(b) for a, b in zip(s, corr)]
    E = len(c)
    if groups and keep < groups:
        per = E // groups
        best = []
        for g in range(groups):
            two = sorted(c[g * per: (g + 1) * per], reverse=True)[:2]
            best.append(two[0] + two[1] if per > 1 and rule == "top2" else two[0])
        kept = sorted(range(groups), key=lambda g: (-best[g], g))[:keep]
        c = [v if i // per in kept else -math.inf for i, v in enumerate(c)]
    order = sorted((i for i in range(E) if c[i] > -math.inf), key=lambda i: (-c[i], i))
    return order[:top], s


@pytest.mark.parametrize("score", ["sigmoid", "softmax", "softmax_chosen"])
@pytest.mark.parametrize("E,top,groups,keep,rule", [(4, 1, 0, 0, "max"), (31, 5, 0, 0, "max"), (32, 32, 0, 0, "max"), (32, 4, 8, 4, "max"),
                                                    (32, 3, 32, 3, "max"), (24, 2, 4, 1, "top2"), (33, 4, 0, 0, "max")])
def test_choice_by_rank(E, top, groups, keep, rule, score):
    from rustinfer_b200.ops import kernels as K
    gen = torch.Generator().manual_seed(E * 7 + top)
    T = 40
    z = torch.randint(-4, 5, (T, E), generator=gen).float() / 2         # many equals
    corr = torch.randint(0, 2, (E,), generator=gen).float() / 4 if score == "sigmoid" else None
    hidden = E - top > 4 and not groups and score != "softmax"
    if hidden:
        z[3, 1] = float("nan")                               # is not chosen
    ids, wts = torch.empty((T, top), dtype=torch.int32, device=DEV), torch.empty((T, top), device=DEV)
    counts = torch.zeros(E, dtype=torch.int32, device=DEV)
    K.moe_route(z.to(DEV), corr.to(DEV) if corr is not None else None, top, groups, keep, score != "softmax_chosen", ids, wts, counts, score=score,
                group_score=rule)
    for t in range(T):
        want, s = rules(z[t], corr if corr is not None else torch.zeros(E), top, groups, keep, score, rule)
        assert ids[t].tolist() == want
        w = s[want].double()
        w = torch.softmax(w, -1) if score == "softmax_chosen" else w / w.sum()
        assert torch.allclose(wts[t].cpu().double(), w, rtol=1e-5, atol=0)        # two exponentials, a sum of 32, a quotient: 2 ulp each
    assert counts.sum().item() == T * top and torch.equal(torch.bincount(ids.flatten().cpu(), minlength=E), counts.cpu().long())
