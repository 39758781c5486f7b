"""The 16-bit copies of fp32 parameters that the layers keep: usable wherever the parameter is."""
import pytest
import torch


def test_copy_made_in_inference_mode_is_an_ordinary_tensor():
    from cubework_b200 import ops
    w = torch.nn.Parameter(torch.randn(8, 8))
    with torch.inference_mode():
        s = ops.shadow(w, torch.bfloat16)
        assert torch.equal(s, w.bfloat16())
    assert not s.is_inference() and not s.requires_grad
    (torch.randn(8, 8).bfloat16().requires_grad_(True) @ s).sum().backward()     # may be saved for a backward pass
    with torch.no_grad():
        w.mul_(2.0)
    assert torch.equal(ops.shadow(w, torch.bfloat16), w.detach().bfloat16())      # and refreshed in place outside
    with torch.no_grad():
        w.mul_(3.0)
    with torch.inference_mode():
        assert torch.equal(ops.shadow(w, torch.bfloat16), w.bfloat16())
    with torch.no_grad():
        w.mul_(0.5)
    s = ops.shadow(w, torch.bfloat16)
    assert torch.equal(s, w.detach().bfloat16()) and not s.is_inference()


@pytest.mark.gpu
@pytest.mark.parametrize("params", ["master", "16bit"])
def test_training_after_evaluation_in_inference_mode(params):
    from cubework_b200 import module as cube_nn
    from cubework_b200.global_vars import env
    env.load(mode=None)
    torch.manual_seed(0)
    with torch.device("cuda"):
        m = torch.nn.Sequential(cube_nn.Linear(64, 128, activation="gelu"), cube_nn.LayerNorm(128), cube_nn.Linear(128, 64))
    if params == "16bit":
        m.bfloat16()
    opt = torch.optim.SGD(m.parameters(), lr=0.1)                 # updates the parameters behind the copies' back
    x = torch.randn(16, 64, device="cuda").bfloat16()

    def forward():
        with torch.autocast("cuda", dtype=torch.bfloat16):
            return m(x)

    for _ in range(2):
        with torch.inference_mode():
            seen = forward()
        y = forward()
        assert torch.equal(y, seen)
        y.float().square().mean().backward()
        assert all(p.grad is not None for p in m.parameters())
        opt.step()
        opt.zero_grad(set_to_none=True)
