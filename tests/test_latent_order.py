"""Where a launch without programmatic dependence stands in a step with prompt portions (no GPU)."""
from __future__ import annotations

import threading


def test_the_mark_for_the_next_launch_is_the_threads_own():
    """Another thread's launch in between does not use it up."""
    from inference_bench_b200.kernels import lib
    core, other = lib.load(), []
    core.ib_set_pdl(1)
    core.ib_pdl_skip_next()
    t = threading.Thread(target=lambda: other.append(core.ib_pdl_enabled()))
    t.start()
    t.join()
    assert other == [1] and core.ib_pdl_enabled() == 0 and core.ib_pdl_enabled() == 1


def _latent_forward(monkeypatch, plan, given=None):
    """The names of what one forward pass of latent attention asks for, in order, with nothing run; `given` collects the named arguments."""
    from types import SimpleNamespace

    import torch

    from inference_bench_b200.kernels import ops
    from inference_bench_b200.parts.latent import LatentAttention
    from inference_bench_b200.parts.standard import NoPositionEncoding
    done, T = [], 40
    for name in ("latent_prepare", "gemm_heads", "latent_attention_mma", "latent_prefill"):
        monkeypatch.setattr(ops, name, lambda *a, _name=name, **kw: (done.append(_name), given is not None and given.append((_name, kw))))
    monkeypatch.setattr(ops, "latent_keys_values", lambda *a, **kw: (done.append("latent_keys_values"), None))
    monkeypatch.setattr(ops, "rows_mma_fits", lambda *a: True)
    rt = SimpleNamespace(act_dtype=torch.bfloat16, sm_count=148, status=None, options=SimpleNamespace(expert_gemm="auto", latent_attention="auto"),
                         empty=lambda shape, dtype=torch.bfloat16: torch.empty(shape, dtype=dtype),
                         linear=lambda x, w, add_to=None: (done.append(f"linear {w}"), torch.empty(1, x.shape[0], 1))[1],
                         next_in_order=lambda ctx: done.append("next_in_order"))
    att = LatentAttention("a", 64, 2, 64, 32, 64, 64, 1.0, 1e-5, NoPositionEncoding())
    att.w_in, att.wo, att.wuk_t, att.wuv, att.w_kv = "in", "out", None, None, object()
    monkeypatch.setattr(att, "_tensor_cores", lambda rt: True)
    monkeypatch.setattr(att, "_slices", lambda ctx, view: (1, 1 << 30))
    monkeypatch.setattr(att, "_rows_and_units", lambda ctx: (16, None))
    monkeypatch.setattr(att, "_expanded", lambda ctx: plan)
    monkeypatch.setattr(att.position, "tables", lambda ctx: (None, None))
    ctx = SimpleNamespace(rt=rt, n_tokens=T, fixed_shape=False, positions=None, seg_of_token=None, seg_start=None, seg_pos0=None, memo={})
    att.forward(ctx, torch.empty(T, 64), SimpleNamespace(c_view=lambda: None))
    return done


def test_the_output_projection_follows_the_prompt_attention_in_order(monkeypatch):
    """The prompt attention of a latent layer holds tensor memory. The output projection behind it must not be left waiting for that while the norm
    after it lets a third product start, so it is launched when everything before it is done; the form without tensor memory needs no such launch."""
    done = _latent_forward(monkeypatch, (None, None, None))
    assert done[-3:] == ["latent_prefill", "next_in_order", "linear out"] and done.count("next_in_order") == 1
    assert "next_in_order" not in _latent_forward(monkeypatch, None)


def test_the_maps_take_the_rows_that_need_them(monkeypatch):
    """Beside portions with keys and values per head, the other tokens' queries alone go to the latents' space and back; without such portions all do."""
    rows = object()
    for plan, want in (((None, None, (16, None, rows)), [rows, rows]), ((None, None, None), []), (None, [None, None])):
        given = []
        _latent_forward(monkeypatch, plan, given)
        assert [kw["rows"] for name, kw in given if name == "gemm_heads"] == want
