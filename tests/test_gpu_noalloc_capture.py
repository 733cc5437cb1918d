"""cup2d_adv_diff_noalloc captured into a CUDA graph after a first call, behind
and ahead of other work of the captured stream, on both sides of the
one-launch rule and with planes that are only 8-byte aligned: every replay
gives the bits of a plain call on the inputs that the planes hold then."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bpdx,bpdy,shift", [(1, 1, 0), (8, 8, 1), (9, 8, 0), (40, 24, 0), (40, 24, 1)])
def test_capture(bpdx, bpdy, shift):
    import torch
    from cubismup_2d_b200 import abi
    from cubismup_2d_b200.synthetic import noise_field
    nx, ny = 32 * bpdx, 32 * bpdy
    n, h = nx * ny, 1.0 / (32 * max(bpdx, bpdy))
    u, v, a, b, c, d = (torch.zeros(n + 2, dtype=torch.float64, device="cuda")[shift:shift + n] for _ in range(6))

    def call(src, dst):
        rc = abi.lib().cup2d_adv_diff_noalloc(src[0].data_ptr(), src[1].data_ptr(), dst[0].data_ptr(),
                                              dst[1].data_ptr(), bpdx, bpdy, h, 3e-4, 2e-3, 0.2, -0.1,
                                              torch.cuda.current_stream().cuda_stream)
        assert rc == abi.OK

    def fill(seed):
        for k, p in enumerate((u, v)):
            p.copy_(torch.from_numpy(np.ascontiguousarray(noise_field(seed, k, ny, nx, amp=1.0)).reshape(-1)))

    def work():                              # two steps between other kernels of the stream
        u.mul_(0.5)
        call((u, v), (a, b))
        call((a, b), (c, d))
        c.add_(1.0)

    fill(51)
    work()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        work()
    for seed in (52, 53):
        fill(seed)
        work()
        want = c.clone(), d.clone()
        fill(seed)
        c.zero_(), d.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(c, want[0]) and torch.equal(d, want[1])
