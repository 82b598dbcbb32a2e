"""Insertions whose spectrum store cannot be allocated: the plan's workspace
without the store serves, the lines are evaluated in the contraction, and the
cube is the one with the store (FP32 form: its bits; else the form's products
of the same lines, at the package's bar of 1e-5 of peak)."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NX, NY, NC, N_PART = 40, 50, 200, 4000


def setup(form, model):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles, InsertionEngine
    eng = InsertionEngine("cuda:0")
    rng = np.random.default_rng(form)
    h = rng.uniform(1.0, 4.0, N_PART)
    parts = DeviceParticles.from_host(
        eng.device, rng.uniform(0, NX, N_PART), rng.uniform(0, NY, N_PART), np.ceil(h), h,
        v=rng.uniform(-350, 350, N_PART), sigma=rng.uniform(20, 60, N_PART),
        amp=rng.uniform(1, 2, N_PART))
    edges = torch.from_numpy(np.arange(NC + 1)[::-1] * 4.0 - NC * 2.0).to(eng.device)
    code = N.MG_SPECTRUM_GAUSSIAN if model == "gaussian" else N.MG_SPECTRUM_DIRAC
    return eng, parts, edges, code, [(N.MG_KERNEL_WENDLAND_C2, 0.0)]


def refuse_above(monkeypatch, limit):
    import torch
    from martini_gb300 import engine
    real = torch.empty
    asked = []

    def empty(*a, **k):
        if k.get("dtype") is torch.uint8 and a[0] > limit:
            asked.append(a[0])
            raise torch.cuda.OutOfMemoryError("no room")
        return real(*a, **k)

    monkeypatch.setattr(engine.torch, "empty", empty)
    return asked


@pytest.mark.parametrize("form", [0, 2, 3], ids=["fp32", "f16x3", "bf16x6"])
@pytest.mark.parametrize("model", ["gaussian", "dirac"])
@pytest.mark.parametrize("batch", [False, True])
def test_without_room_for_the_store(form, model, batch, monkeypatch):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import InsertionEngine, insert_batch
    eng, parts, edges, code, table = setup(form, model)

    def insert(e):
        if not batch:
            return e.insert(parts, table, code, 0.0, NX, NY, NC, edges, form=form)[0]
        item = dict(parts=parts, edges=edges, nx=NX, ny=NY, nc=NC)
        return insert_batch(e, [item, item], table, code, form=form)[1][0]

    want = insert(eng)
    cube = torch.empty((NX, NY, NC), device=eng.device)
    prob = eng.problem(parts, table, code, 0.0, NX, NY, NC, 0, 0, edges, cube, None, form)
    both = (N.Problem * 2)(prob, prob)
    k = 2 if batch else 1
    base, need = C.c_size_t(), C.c_size_t()
    N.check(eng.lib.mg_workspace_size_batched(both, k, 0, 0, C.byref(base)))
    ws, info = torch.empty(base.value, dtype=torch.uint8, device=eng.device), N.PlanInfo()
    N.check(eng.lib.mg_plan_batched(both, k, C.c_void_p(ws.data_ptr()), base.value, None,
                                    C.byref(info)))
    N.check(eng.lib.mg_workspace_size_batched(both, k, info.n_pairs, info.n_partial_items,
                                              C.byref(need)))
    assert need.value < info.workspace_bytes
    asked = refuse_above(monkeypatch, need.value)
    got = insert(InsertionEngine("cuda:0"))
    assert asked == [info.workspace_bytes]
    if form == 0:
        assert torch.equal(got, want)
    else:
        assert (got - want).abs().max() <= 1e-5 * want.abs().max()
