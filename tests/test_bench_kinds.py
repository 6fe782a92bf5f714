"""The benchmark's kinds of kernel know every entry point of latent attention and of the float32 portions (no GPU)."""
import sys
from pathlib import Path

import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))


@pytest.mark.parametrize("design,kind,entries", [
    *[(d, k, ["ib_latent_attention", "ib_latent_attention_mma", "ib_latent_gather", "ib_gemm_bf16_2cta", "ib_latent_prefill"])
      for d, k in (("zabonex", "attention"), ("ditalorn", "attention"), ("gokosun", "latent"))],
    *[(d, "attention", ["ib_attention_generic", "ib_attention_prompt_f32"]) for d in ("busadra", "lulenex", "fedipel", "gokosun")]])
def test_kinds(design, kind, entries):
    import bench
    assert set(entries) <= set(bench.DESIGN_KINDS[design][kind])
