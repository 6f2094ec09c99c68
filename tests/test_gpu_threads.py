"""Contexts of several host threads on one device."""
import threading

import numpy as np
import pytest

from atrip_gb300 import capi, synth

pytestmark = pytest.mark.gpu
NAMES = ("epsi", "epsa", "Tai", "Tabij", "Vabij", "Vijka", "Vabci")


# systems whose launches of one kernel ask for different shared memory, so that
# a thread that set the kernel's limit to its own size would fail the others'
@pytest.mark.parametrize("form,slices,variant", [("fp64", 0, 0), ("split_f16", 2, 0),
                                                 ("split_f16", 2, 2), ("split_bf16", 3, 1)])
def test_contexts_of_different_sizes(form, slices, variant):
    bad = []

    def work(No, Nv, n):
        try:
            d = synth.make_inputs(No, Nv, No)
            with capi.Context(No, Nv, 0) as ctx:
                for k in NAMES:
                    ctx.upload(k, d[k])
                ctx.set_tuning(split_variant=variant)
                kw = dict(form=form, slices=slices, use_j=False, max_iterations=20)
                ref = ctx.run(**kw)
                for _ in range(n):
                    if ctx.run(**kw).energy != ref.energy:
                        raise AssertionError("another energy")
        except Exception as e:  # noqa: BLE001 - reported below
            bad.append((No, str(e)))

    threads = [threading.Thread(target=work, args=a)
               for a in ((8, 40, 2000), (16, 33, 2000), (24, 30, 2000))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
