"""Batches of one composition in turn, with other frames in other buffers each
time, through every choice of graphs and stage fusion: a replay must not hold on
to the first batch's."""
import numpy as np
import pytest

import oracle
from vaco_b200 import synth
from vaco_b200.gpu import Context, DeviceFrame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("fusion", [0, 1])
def test_other_frames_in_other_buffers(graphs, fusion, oracle_threads):
    import torch

    ctx = Context(0)
    ctx.set_tuning(use_graphs=graphs, stage_fusion=fusion)
    stream = torch.cuda.Stream()
    kept = []  # the first batches' buffers stay allocated
    for i in range(3):
        frames = [synth.make_small(10 * i + k, w, h, bd, upscaled_width=up, with_lvl_map=i == 1)
                  for k, (w, h, bd, up) in enumerate([(200, 136, 10, None), (328, 200, 8, 400)])]
        if i == 2:
            frames[0].deblock_levels = (0, 0, 0, 0)  # fewer launches in the per-stage form
        devs = [DeviceFrame(f) for f in frames]
        kept.append(devs)
        torch.cuda.synchronize()
        status, _ = ctx.postfilter_batch_dev(devs, stream=stream.cuda_stream)
        assert status == [0, 0]
        for f, d in zip(frames, devs):
            want, m = oracle.postfilter_frame(f, threads=oracle_threads)
            assert m == 0
            for k, (g, w) in enumerate(zip(d.outputs_numpy(), want)):
                assert np.array_equal(g, w), f"batch {i} plane {k}"
    ctx.close()
