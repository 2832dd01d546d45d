"""Guide inference in its two forms, four whole operands per SM or six in two parts: a row's outputs do
not depend on the batch around it, to the bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LO, HI = np.array([-2.0, 0.0, -2.0], np.float32), np.array([2.0, 2.5, 2.0], np.float32)


@pytest.mark.parametrize("extra", [0, 1, 127])
@pytest.mark.parametrize("tiles_per_sm", [1, 4, 5, 6, 7, 8, 9, 13])
def test_rows_do_not_depend_on_the_batch(core, gpu_ctx, tiles_per_sm, extra):
    import torch

    B = torch.cuda.get_device_properties(0).multi_processor_count * 128 * tiles_per_sm + extra
    g = torch.Generator(device="cuda").manual_seed(B)
    unit = lambda: torch.nn.functional.normalize(torch.randn(B, 3, generator=g, device="cuda"))
    lo, hi = torch.from_numpy(LO).cuda(), torch.from_numpy(HI).cuda()
    q = torch.cat([lo + (hi - lo) * torch.rand(B, 3, generator=g, device="cuda"), unit(), unit()], 1).contiguous()
    u, wi = torch.rand(B, 3, generator=g, device="cuda"), unit().contiguous()
    pdf = torch.rand(B, generator=g, device="cuda")
    net = core.Guide(gpu_ctx, LO, HI, learning_rate=1e-2, seed=3)
    raw, dirs, density, mixed = net.eval(q), *net.sample(q, u), net.pdf(q, wi, pdf)
    for a in (0, B // 2 + 1, B - 777):  # a few tiles by themselves, the last row among them
        s = slice(a, a + 777)
        cut = lambda x: x[s].contiguous()
        assert torch.equal(raw.view(B, -1)[s], net.eval(cut(q)).view(777, -1))
        d, p = net.sample(cut(q), cut(u))
        assert torch.equal(dirs.view(B, 3)[s], d.view(-1, 3)) and torch.equal(density.view(-1)[s], p.view(-1))
        assert torch.equal(mixed.view(-1)[s], net.pdf(cut(q), cut(wi), cut(pdf)).view(-1))
    net.close()
