"""What cavity_loss has the adjoint forward record: states for a tau gradient,
points for the others, nothing where no backward sweep can follow (no_grad, or
no control that requires a gradient)."""
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("grad", [True, False])
@pytest.mark.parametrize("lid_grad", [True, False])
@pytest.mark.parametrize("tau_grad", [True, False])
def test_recorded(monkeypatch, grad, lid_grad, tau_grad):
    from lbmcl_gb300 import adjoint
    made = []

    class Lattice:
        def __init__(self, dim, **kw):
            made.append(kw)

        def adjoint_set_loss(self, *a):
            pass

        def adjoint_forward(self, *a):
            return 0.25

        def close(self):
            pass

    monkeypatch.setattr(adjoint.capi, "Lattice", Lattice)
    lid = torch.full((8, 8), 0.05, requires_grad=lid_grad)
    tau = torch.tensor(0.53, requires_grad=tau_grad)
    with torch.set_grad_enabled(grad):
        loss = adjoint.cavity_loss(lid, tau, None, dim=8, iterations=4, plane_y=4)
    assert loss.item() == 0.25 and loss.requires_grad == (grad and (lid_grad or tau_grad))
    (kw,) = made
    full, tail = bool(kw.get("adjoint_full_states", False)), kw.get("adjoint_tail_segments", 0)
    if not loss.requires_grad:
        assert not full and tail == -1
    else:
        assert full == tau_grad and tail == 0
