"""GPU parity of the BF16 head at the edges of its tiles: one tile, tiles of 8 rows, a last tile that the tensor ends in, one row
more than a full round of 128-row tiles, more stages than the ring holds, the widest row; every token count's first and last row.
Bound as for the head elsewhere: |error| <= 2e-7 * |w| * |x| against fp64."""
import pytest

from augur_v100_b200 import host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,tokens", [(16, 64, 1), (1200, 128, 8), (4096, 6336, 3), (18944, 192, 2), (18960, 832, 5), (37904, 64, 7)])
def test_head_tiles(rows, cols, tokens):
    import torch
    torch.cuda.set_device(0)
    device = torch.device("cuda", 0)
    stream = host.Stream(0)
    generator = torch.Generator(device=device)
    generator.manual_seed(rows + cols)
    weight = torch.randn((rows, cols), device=device, generator=generator).to(torch.bfloat16)
    x = torch.randn((tokens, cols), device=device, generator=generator) * 2.0 ** torch.randint(-9, 9, (tokens, cols), device=device, generator=generator)
    guard = torch.full((tokens * rows + 64,), float("nan"), device=device)
    out = guard[32:32 + tokens * rows].view(tokens, rows)
    torch.cuda.synchronize()
    head = host.Bf16Head.bind(stream, weight, x, out)
    for _ in range(2):
        head.submit()
    stream.synchronize()
    want = x.double() @ weight.double().T
    bound = 2e-7 * x.double().norm(dim=1, keepdim=True) * weight.double().norm(dim=1)
    assert bool(((out.double() - want).abs() <= bound).all())
    assert bool(torch.isnan(guard[:32]).all()) and bool(torch.isnan(guard[32 + tokens * rows:]).all())
    stream.close()
