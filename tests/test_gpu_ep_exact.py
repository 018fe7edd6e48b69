"""GPU: an expert-parallel rank at nine and more assignments per expert on banks of 4-bit codes: it takes the forms that the unsplit layer
takes (the exact grouped product for gate/up and down, 16-bit and fp32 rows), so split and unsplit differ by the order of the fp32 partial
sums only. The decode kernels on either side would show: they round the activations to 15 bits (2e-4)."""
import pytest

from test_gpu_ep import run_split, run_split_a2a
from tqllm_b200 import synth
from util import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("act_dtype", ("bf16", "f32"))
@pytest.mark.parametrize("types,gating,shared,T", (((12, 12, 12), 2, False, 24), ((21, 21, 21), 1, True, 36)))
def test_split_equals_unsplit(types, gating, shared, T, act_dtype):
    shape = synth.LayerShape("ep-exact", 512, 16, 4, 256, gating=gating, sel_bias=gating == 2, shared=shared, types=types, act_dtype=act_dtype)
    got, want = run_split(shape, 16, T, 2, 31 + T)               # 12 and 18 assignments per expert
    assert rel_err(got, want) <= 1e-5
    got, want, _ = run_split_a2a(shape, 16, T, 2, 41 + T)
    assert rel_err(got, want) <= 1e-5
