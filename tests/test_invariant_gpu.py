"""`EngineOptions.invariant` in the designs that are walked from Python: a position's logits are the same bits however its request was
cut and whatever else was in the step (the reference's rule, src/backends/backend.hpp:141-150)."""
import importlib

import numpy as np
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["decay", "delta", "scaled", "delta_channel", "channel"])
@pytest.mark.parametrize("D", [20, 128, 300])
def test_invariant_recurrences_do_not_depend_on_the_cutting(form, D):
    """Fifty rows at once and in portions of nine, sixteen, one, eight and sixteen: the same outputs and the same state, bit for bit."""
    import types
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(D)
    rows, H, V = 50, 3, 17
    make = lambda *shape: torch.randn(*shape, generator=g).cuda()
    q, k, v, beta, skip = make(rows, H * D), make(rows, H * D) * D ** -0.5, make(rows, H * V), make(rows, H).sigmoid(), make(H)
    gate = 0.7 + 0.3 * torch.rand(rows, H * (D if "channel" in form else 1), generator=g).cuda()
    options = {"decay": dict(decay=torch.rand(H, generator=g).cuda()), "channel": dict(gate=gate)}.get(form, dict(gate=gate, beta=beta))
    if form == "scaled":
        options["skip"] = skip
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device="cuda")
    results = []
    for portions in ([rows], [9, 16, 1, 8, 16]):
        state, out, at = torch.zeros(2, H * V * D, device="cuda"), torch.empty(rows, H * V, device="cuda"), 0
        for i, n in enumerate(portions):
            step = types.SimpleNamespace(row_start=i32(0), row_count=i32(n), history=i32(at), state_slots=i32(i % 2), state_slots_out=i32(1 - i % 2),
                                         requests=1, max_row_count=n, rows=n)
            s = slice(at, at + n)
            cut = {key: x[s] if key in ("gate", "beta") else x for key, x in options.items()}
            ops.linear_recurrence(q[s], k[s], v[s], state, step, out[s], H, H, D, V, form=form, invariant=True, **cut)
            at += n
        results.append((out, state[len(portions) % 2].clone()))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("design", ["buzetar", "zamizen", "kisepel", "nomutar", "fipadra", "dikusun"])
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_invariant_schedules_give_a_row_the_same_bits_in_any_batch(tmp_path, design, dtype):
    """The whole model of each design's own tests (every mixer, recurrences among them): prompts whole, with their last rows
    decoded, in portions and mixed with other requests, in runs on both sides of every length at which a kernel has another form."""
    from llmx_b200.engine import Engine, EngineOptions
    tests = importlib.import_module(f"test_{design}_gpu")
    cfg = tests.MODEL_P
    tests.make_folder(str(tmp_path), cfg, 5, dtype=getattr(torch, dtype))
    requests = {f"i{i}": helpers.random_ids(cfg["vocab"], n, seed=80 + i) for i, n in enumerate([70, 9, 40, 33, 81])}
    base = None
    for make in tests.CUTTINGS:
        steps = make(requests)
        engine = Engine.from_dir(str(tmp_path), EngineOptions(dtype=dtype, kv_tokens=helpers.tokens_needed(steps), page_size=4, max_requests=4,
                                                              invariant=True))
        got = helpers.run_trace(engine, steps)
        del engine
        base = base or got
        assert got.keys() == base.keys()
        moved = [k for k in base if not np.array_equal(base[k], got[k])]
        assert not moved, (make.__name__, len(moved), moved[:5])
