"""First-order walks at the sizes where the launch changes shape (half-full warps up to two blocks per SM, full ones
past that, as many blocks on every SM, more walks than lanes): rows against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("app,length", [(0, 7), (2, 9)])
def test_rows_at_every_launch_shape(app, length):
    import torch
    from bingo_b200 import BATCHED, PLAIN, Graph, WalkJob, gen
    from oracle import pyoracle as po
    n = 1 << 11
    src, dst = gen.rmat(11, 8, seed=3)
    w = gen.weights(len(src), gen.W_UNIFORM, 1, 1 << 16, seed=4)
    ex = po.ExactGraph(n)
    ex.load(src, dst, w)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    with Graph(device=0, node2vec=False) as g:
        g.load_edges(src, dst, w, n)
        for k in (127, 128, 129, sms * 128, 2 * sms * 128 - 1, 2 * sms * 128, 2 * sms * 128 + 1, 2 * sms * 256 - 3,
                  2 * sms * 256, 2 * sms * 256 + 1, 3 * sms * 256, 3 * sms * 256 + 5, 4 * sms * 256 - 1,
                  4 * sms * 256 + 1, 5 * sms * 256 + 77):
            starts = (np.arange(k, dtype=np.uint64) * 2654435761 % n).astype(np.uint32)
            want = ex.walk(app, length, starts, seed=k, stop=0.2)
            dev = torch.from_numpy(starts.view(np.int32)).cuda()
            for mode in (PLAIN, BATCHED):
                out = torch.full((k, length), -9, dtype=torch.int32, device="cuda")
                g.walk_jobs([WalkJob(app=app, length=length, starts=dev, n_starts=k, seed=k, stop_prob=0.2, out=out)],
                            mode=mode)
                assert np.array_equal(out.cpu().numpy(), want), (k, mode)
