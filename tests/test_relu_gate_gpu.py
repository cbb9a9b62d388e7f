"""ReLU's gradient where the pre-activation is positive but far below what half precision resolves: with weight 1e-9
and bias 1e-8 every pre-activation lies between 4e-9 and 2e-8, so ReLU is the identity and must have its gradients,
bit for bit, on every launch plan and in both layouts."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plan", ["auto", "fused", "twopass", "wave", "resident", "channels_first"])
@pytest.mark.parametrize("shape", [(2, 1000, 64, 8), (1, 700, 80, 8)], ids=str)  # vectors inside one group / across groups
def test_positive_pre_activations_keep_their_gradient(shape, plan, monkeypatch):
    import channels_last_groupnorm_b200  # noqa: F401

    if plan not in ("auto", "channels_first"):
        monkeypatch.setenv("GNB200_FORCE_PATH", plan)
    N, R, C, G = shape
    torch.manual_seed(2)
    make = lambda: torch.randn(N, R, C, device="cuda").clamp_(-4, 4).bfloat16().permute(0, 2, 1)
    x, dy = make(), make()
    if plan == "channels_first":
        x, dy = x.contiguous(), dy.contiguous()
    w, b = (torch.full((C,), v, device="cuda", dtype=torch.bfloat16) for v in (1e-9, 1e-8))
    y, mean, rstd = torch.ops.gnb200.fwd(x, w, b, G, 1e-5, 1)
    assert (y > 0).all()
    relu = torch.ops.gnb200.bwd_f32(dy, x, w, b, mean, rstd, G, 1)
    identity = torch.ops.gnb200.bwd_f32(dy, x, w, b, mean, rstd, G, 0)
    for a, c in zip(relu, identity):
        assert c.abs().max() > 0 and torch.equal(a, c)
