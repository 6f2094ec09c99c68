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


@pytest.mark.parametrize("form,S,sizes,kernel", [
    ("split_f16", 2, [(12, 12), (20, 9)], "split"), ("split_f16", 2, [(11, 12), (11, 13)], "tensor_core"),
    ("split_f16", 2, [(11, 12), (20, 12)], "tensor_core"), ("split_f16", 2, [(3, 5), (28, 20)], "split"),
    ("split_f16", 2, [(12, 199)], "split"), ("split_f16", 2, [(12, 200)], "tensor_core"),
    ("split_bf16", 3, [(16, 12), (16, 14)], "split"), ("split_bf16", 3, [(16, 12), (17, 14)], "tensor_core"),
    ("split_bf16", 3, [(29, 8)], "tensor_core"), ("split_bf16", 4, [(16, 12)], "tensor_core")])
def test_batches(form, S, sizes, kernel):
    ctxs = [_ctx(*s) for s in sizes]
    with capi.Batch(ctxs) as b:
        got = b.run(form=form, slices=S, use_j=False, max_iterations=99)
        assert {c.last_kernel() for c in ctxs} == {kernel}
    for c, r in zip(ctxs, got):
        one = c.run(form="fp64", use_j=False, max_iterations=99)
        assert abs(r.energy - one.energy) <= 1e-3 * abs(one.energy)  # the split forms': 1e-5 or less
        c.close()
