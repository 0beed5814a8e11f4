"""Who decides the launch of a batch of a few points: the caller where the caller gave it, the tuner where
it measured these counts, and the tuner's pairs at every other count of a tuned batch."""
import pytest

from tests.test_gpu_batch import check, setup

pytestmark = pytest.mark.gpu

FEW, OTHER = [2, 3, 1, 4], [5, 1, 7, 2]


def launch(b):
    n = len(b.plans)
    return b.launches, [b.plan_blocks_per_sm(k) for k in range(n)], [b.lanes_per_point(k) for k in range(n)]


def run(b, out, want):
    import torch

    for o in out:
        o.fill_(float("nan"))
    b.run()
    torch.cuda.synchronize()
    check(out, want)


@pytest.mark.parametrize("plans", [slice(0, 1), slice(0, 4)])
def test_a_tuned_batch_keeps_its_pairs_at_counts_that_were_not_timed(plans):
    from pacuda_b200 import batch as B

    large, few = [[x[plans] for x in setup("f64", c)] for c in ([3000, 800, 900, 700], FEW)]
    b = B.Batch(*large[:3])
    b.tune()
    tuned = launch(b)
    b.update(few[1], FEW[plans], few[2])
    assert launch(b) == tuned
    run(b, few[2], few[3])


def test_a_measurement_is_of_its_counts():
    from pacuda_b200 import batch as B

    first, second = setup("f64", FEW), setup("f64", OTHER)
    b = B.Batch(*first[:3])
    b.tune()
    there = launch(b)
    b.update(second[1], OTHER, second[2])
    pairs = launch(b)  # the tuned pairs
    run(b, second[2], second[3])
    b.update(first[1], FEW, first[2])
    assert launch(b) == there
    run(b, first[2], first[3])
    b.set_plan_blocks_per_sm(0, 2)
    b.set_plan_blocks_per_sm(0, 0)  # no longer what was measured
    assert launch(b)[1][1:] == pairs[1][1:]
    run(b, first[2], first[3])


def test_one_block_per_sm_that_the_caller_gave():
    from pacuda_b200 import batch as B

    plans, ext, out, want = setup("f64", FEW)
    b = B.Batch(plans, ext, out)
    spread = launch(b)
    assert spread == (1, [1] * 4, [512] * 4)
    b.blocks_per_sm = 1
    given = launch(b)
    assert given[2] == [p.lanes_per_point for p in plans] != spread[2]
    run(b, out, want)
    b.blocks_per_sm = 0
    assert launch(b) == spread
    run(b, out, want)
