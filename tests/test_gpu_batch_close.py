"""A batch plan closed right after a run on a caller's stream: its buffers go back
when the run has ended, whatever takes them next."""
import pytest

pytestmark = pytest.mark.gpu


def test_close_after_run(gpu):
    import torch

    from compmatmul_b200.batch import BatchPlan
    g = torch.Generator(device="cuda").manual_seed(4)
    mats = [(torch.randn((2000, 3000), device="cuda", generator=g), torch.randn((2000, 2900), device="cuda", generator=g))
            for _ in range(4)]

    def plan(seed):
        return BatchPlan([dict(AT=a, B=b, d=7, b=1 << 14, seed=seed + i, variant=("fft", "fwht")[i % 2])
                          for i, (a, b) in enumerate(mats)], f32=True, tune=False, dense=False)

    want = plan(1)
    want.run()
    torch.cuda.synchronize()
    want_p = [q["p"].clone() for q in want.products]
    want.close()
    stream = torch.cuda.Stream()
    for _ in range(3):
        first = plan(1)
        first.run(stream)
        first.close()
        second = plan(9)  # takes the first one's memory, on a stream of its own
        second.run()
        second.close()
        torch.cuda.synchronize()
        for q, p in zip(first.products, want_p):
            assert torch.equal(q["p"], p)
