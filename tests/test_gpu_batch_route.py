"""Whether a batch plan's products take the product sketch: not where so few do that
its launches cost more than their transforms (measured on B200: 1.2 to 2.8 times),
but the same products do in a plan of many."""
import pytest

pytestmark = pytest.mark.gpu

# (variant, f32, n_a, n_inner, n_b, b, d), products up to which the transforms are faster
SHAPES = [(("fft", True, 500, 100, 500, 4096, 7), 2), (("fwht", True, 500, 100, 500, 4096, 7), 4),
          (("fwht", False, 256, 256, 256, 2048, 5), 2), (("fwht", True, 1000, 64, 1000, 16384, 5), 2)]


@pytest.mark.parametrize("shape,few", SHAPES)
def test_few_and_many(gpu, shape, few):
    import torch

    from compmatmul_b200.batch import BatchPlan
    variant, f32, n_a, k, n_b, b, d = shape
    dt = torch.float32 if f32 else torch.float64
    g = torch.Generator(device="cuda").manual_seed(2)
    A, B = (torch.randint(-9, 10, (k, n), device="cuda", generator=g).to(dt) for n in (n_a, n_b))
    tiles = -(-n_a // 256) * -(-n_b // 256) * (8 if f32 else 15)
    sketches = {}
    for count in (1, few, 32):
        plan = BatchPlan([dict(AT=A, B=B, d=d, b=b, seed=5, variant=variant)] * count, f32=f32, tune=False, dense=False)
        assert (plan.info()["items"] == count * tiles) == (count == 32), (count, plan.info())
        plan.run()
        torch.cuda.synchronize()
        sketches[count] = plan.products[-1]["p"].clone()
        plan.close()
    want = sketches[32]  # (exact: integers)
    assert torch.equal(want, want.round())
    for count in (1, few):
        assert (sketches[count] - want).abs().max() <= (2e-5 if f32 else 1e-11) * want.abs().max()
