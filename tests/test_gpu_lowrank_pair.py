"""K and V through projection and reconstruction in one kernel, against an fp32 reference with the latent in bf16."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# row counts around the 128-row item and its 32-row stores and with several items per CTA; widths with a ragged
# 64-column k block and output chunk; every rank the kernel takes; fp32, bf16 and no biases
@pytest.mark.parametrize("M,K,R,N,bias", [(1, 64, 16, 64, "f32"), (127, 72, 32, 1000, "bf16"), (161, 1000, 48, 72, "none"),
                                          (4099, 1024, 64, 1024, "bf16"), (20000, 256, 64, 4096, "f32"),
                                          (38401, 128, 16, 192, "f32")])
def test_lowrank_pair_matches_reference(M, K, R, N, bias):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pikv_b200
    from pikv_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(M)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")   # noqa: E731
    xs = [randn(M, K).bfloat16() for _ in range(2)]
    w1 = [(randn(R, K) / K ** 0.5).bfloat16() for _ in range(2)]
    w2 = [(randn(N, R) / R ** 0.5).bfloat16() for _ in range(2)]
    dt = {"f32": torch.float32, "bf16": torch.bfloat16, "none": None}[bias]
    b1 = [None if dt is None else randn(R).to(dt) for _ in range(2)]
    b2 = [None if dt is None else randn(N).to(dt) for _ in range(2)]
    outs = ops.lowrank_pair(xs, w1, b1, w2, b2)
    torch.cuda.synchronize()
    assert pikv_b200.lib().pikv_lowrank_error_state() == 0
    for i in range(2):
        z = xs[i].double() @ w1[i].double().T + (0 if dt is None else b1[i].double())
        z = torch.relu(z).bfloat16().double()
        y = z @ w2[i].double().T + (0 if dt is None else b2[i].double())
        # bf16 has 8 significant bits: its unit roundoff is 2^-8 of |y|, and a latent next to a rounding boundary may fall
        # to the other side, two roundoffs or 2^-7 of it times its weight, allowed for every one of the R terms
        terms = z.abs() @ w2[i].double().T.abs()
        err = (outs[i].double() - y).abs()
        assert bool((err <= y.abs() * 2.0 ** -8 + terms * 2.0 ** -7 + 1e-6).all())
        assert float(err.norm() / y.norm()) < 2.0 ** -8
