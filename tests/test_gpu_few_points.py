"""Batches of a few points: up to one point per SM in all plans together, a batch runs one point per
block and one block per SM; past that, and wherever the caller gives the launch, its other choices.
The counts lie on both sides of that line, alone and as several plans, and an update crosses it in
both directions (also on a tuned and on a captured batch). Every output has the oracle's bits."""
import pytest

from tests.test_gpu_batch import check, setup

pytestmark = pytest.mark.gpu


def sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("kind", ["f64", "df64", "mixed"])
@pytest.mark.parametrize("over", [None, 0, 1])
def test_counts_around_one_point_per_sm(kind, over):
    from pacuda_b200 import batch as B
    import torch

    counts = [1, 1, 1, 1] if over is None else [sms() - 40 + over, 7, 32, 1]
    plans, ext, out, want = setup(kind, counts)
    b = B.Batch(plans, ext, out)
    b.blocks_per_sm = 0
    few = sum(counts) <= sms()
    assert not few or (b.launches == 1 and all(b.plan_blocks_per_sm(k) == 1 for k in range(4)))
    for tuned in (False, True):
        if tuned:
            b.tune()
        b.run()
        torch.cuda.synchronize()
        check(out, want)
    assert not few or b.launches == 1


def test_an_update_crosses_the_line_both_ways():
    from pacuda_b200 import batch as B
    import torch

    large, small = setup("f64", [300, 33, 129, 5]), setup("f64", [2, 3, 1, 4])
    b = B.Batch(*large[:3])
    b.blocks_per_sm = 0
    launches = b.launches
    for plans, ext, out, want in (large, small, large, small):
        for o in out:
            o.zero_()
        counts = [int(e.numel() // (4 * p.template.external_count)) for p, e in zip(plans, ext)]
        b.update(ext, counts, out)
        assert b.launches == (1 if sum(counts) <= sms() else launches)
        b.capture()
        b.run()
        torch.cuda.synchronize()
        check(out, want)


def test_a_given_choice_stays():
    from pacuda_b200 import batch as B
    import torch

    plans, ext, out, want = setup("f64", [2, 3, 1, 4])
    b = B.Batch(plans, ext, out)
    b.blocks_per_sm = 2
    assert all(b.plan_blocks_per_sm(k) == 2 for k in range(4))
    b.blocks_per_sm = 0
    b.set_plan_blocks_per_sm(1, 4)
    assert b.plan_blocks_per_sm(1) == 4
    b.run()
    torch.cuda.synchronize()
    check(out, want)
