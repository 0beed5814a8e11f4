"""The pinned descriptor block of a batch has one reader on the device that runs late: the copy of a
queued run or replay. Whatever writes the block again (an update, the launch's choices) waits for it."""
import pytest

from tests.test_gpu_batch import check, setup

pytestmark = pytest.mark.gpu

LARGE, SMALL = [300, 33, 129, 5], [2, 3, 1, 4]  # (in all: above one point per SM and below)


def change(b, how, other):
    plans, ext, out, want = other
    if how == "update":
        b.update(ext, SMALL, out)
    elif how == "blocks":
        b.blocks_per_sm = 2
    elif how == "plan blocks":
        b.set_plan_blocks_per_sm(0, 4)
    else:
        b.tune()


@pytest.mark.parametrize("captured", [True, False])
@pytest.mark.parametrize("how", ["update", "blocks", "plan blocks", "tune"])
def test_a_queued_run_keeps_its_descriptors(how, captured):
    import torch

    from pacuda_b200 import batch as B

    first, other = setup("f64", LARGE), setup("f64", SMALL)
    b = B.Batch(*first[:3])
    b.blocks_per_sm = 0
    if captured:
        b.capture()
    b.run()  # (what loads kernels and modules has run)
    torch.cuda.synchronize()
    for o in first[2]:
        o.fill_(float("nan"))
    queued = torch.cuda.Event()
    torch.cuda._sleep(200_000_000)  # about a tenth of a second on the stream, ahead of the run's copy
    b.run()
    queued.record()
    assert not queued.query()
    change(b, how, other)
    # before anything else: the queued run's outputs are its own (tune times its launches into them)
    if how != "tune":
        queued.synchronize()
        check(first[2], first[3])
    b.run()
    torch.cuda.synchronize()
    check(first[2], first[3])
    if how == "update":
        check(other[2], other[3])
