"""What the creation of a batched sweep prepares: the form that will run, and nothing of the other."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def sweep(form):
    from lentils_gb300.sweep import BatchedSweep, draw_samples

    class Fixed:
        tuned = 0

        def params(self, *a):
            return 16, 1024
    samples = draw_samples(np.random.default_rng(3), 3, sizes=(128,), nvis_range=(2e4, 4e4))
    return BatchedSweep(samples, tuner=Fixed(), form=form)


def test_statistics_are_of_the_form_that_runs(native):
    """CTAs and shared memory of the kernels that a run launches: every item once in a gridding and
    once in a degridding kernel, a CTA per pixel chunk, the zeroing; the persistent kernel's
    resident slots at most."""
    split, persistent = sweep(0), sweep(1)
    a, b = split.stats(), persistent.stats()
    assert a["nwork"] == b["nwork"] and a["total_vis"] == b["total_vis"]
    assert a["blocks"] == a["nwork"] + 16 * 3
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert 1 <= b["blocks"] <= min(b["nwork"], 2 * sms)
    assert 0 < a["smem_bytes"] < b["smem_bytes"]
    for s in (split, persistent):
        s.run()
        s.stream.synchronize()
    for x, y in zip(split.vis_out, persistent.vis_out):
        assert torch.equal(x, y)
