"""CPU: what the layer call refuses, and how, before anything touches a device."""
import pytest
import torch


def _params(E=1):
    p = {n: torch.zeros(64 * E, 256, dtype=torch.bfloat16) for n in ("gate_weight", "up_weight", "down_weight")}
    p["router"] = torch.zeros(4, 64, E, dtype=torch.bfloat16)
    return p


@pytest.mark.parametrize("proj", [False, True])
def test_cpu_tensors_are_a_type_error(proj):
    import flashmhf_b200 as fm
    p = _params()
    if proj:
        p.update(w_self=torch.zeros(256, 256, dtype=torch.bfloat16), w_self_2=torch.zeros(256, 256, dtype=torch.bfloat16))
    with pytest.raises(TypeError):
        fm.mhffn_layer(torch.zeros(1, 4, 256, dtype=torch.bfloat16), p, H=4, Hkuv=4, E=1, apply_rmsnorm=False)


@pytest.mark.parametrize("E", [2, 4, 32])
def test_a_router_of_another_number_of_sub_networks_is_refused(E):
    import flashmhf_b200 as fm
    with pytest.raises(ValueError):
        fm.mhffn_layer(torch.zeros(1, 4, 256, dtype=torch.bfloat16), _params(1), H=4, Hkuv=4, E=E, apply_rmsnorm=False)
