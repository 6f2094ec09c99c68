"""The kernel that a call without launch parameters takes, where the better one
changes with the sizes (csrc/split.cuh, csrc/batch.cu)."""
import pytest

from atrip_gb300 import capi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _ctx(No, Nv):
    ctx = capi.Context(No, Nv, 0)
    g = torch.Generator(device="cuda").manual_seed(No)
    for k, n in (("epsi", No), ("epsa", Nv), ("Tai", No * Nv), ("Tabij", (No * Nv) ** 2),
                 ("Vabij", (No * Nv) ** 2), ("Vijka", No ** 3 * Nv), ("Vabci", Nv ** 3 * No)):
        t = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
        if k.startswith("eps"):
            t = (1 + t.abs()) * (1 if k == "epsa" else -1)
        torch.cuda.synchronize()
        ctx.upload(k, t)
    del t
    torch.cuda.empty_cache()
    return ctx


@pytest.mark.parametrize("No,Nv,kernel", [(11, 20, "tensor_core"), (12, 20, "split"), (52, 12, "split"),
                                          (53, 12, "tensor_core"), (56, 12, "tensor_core"),
                                          (57, 12, "split"), (54, 384, "tensor_core"),
                                          (54, 385, "split")])
def test_two_fp16_slices(No, Nv, kernel):
    with _ctx(No, Nv) as ctx:
        ctx.run(form="split_f16", use_j=False, max_iterations=9)
        assert ctx.last_kernel() == kernel


@pytest.mark.parametrize("No,kernel", [(56, "tensor_core"), (57, "split"), (64, "split")])
def test_four_bf16_slices(No, kernel):
    with _ctx(No, 12) as ctx:
        ctx.run(form="split_bf16", slices=4, use_j=False, max_iterations=9)
        assert ctx.last_kernel() == kernel
