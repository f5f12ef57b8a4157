"""On a B200: groups of one or two rows, which either kernel of a few rows takes, by the layer's types, its row lengths and the
call's assignments. Which one ran shows in the bits: the integer-dot kernels sum a row as they do in a layer kept off the
tensor cores, the other kernel in its own order."""
import numpy as np
import pytest

from c0ven_b200 import MoELayer, synth
from test_gpu_parity import MAX_REL, TYPES, check

pytestmark = pytest.mark.gpu

HEAVY = {synth.Q4_K, synth.Q6_K, synth.IQ4_XS, synth.IQ4_NL}
CODEBOOK_OF_FOUR = {synth.IQ3_S, synth.IQ3_XXS}


def by_integer_dots(gate, down, assignments):
    if gate in HEAVY and down in HEAVY:
        return assignments < 32
    return assignments < 200 or gate == synth.IQ3_S or (gate == synth.Q8_0 and down in CODEBOOK_OF_FOUR)


@pytest.mark.parametrize("gate", TYPES)
@pytest.mark.parametrize("down", TYPES)
def test_rows_of_the_specialised_lengths(gate, down):
    layer = synth.make_layer(n_embd=512, n_ff=256, n_experts=512, n_used=10, gate_type=gate, down_type=down, shexp_gate_type=synth.Q8_0,
                             shexp_down_type=synth.Q8_0, seed=gate * 43 + down)
    for k in ("gate_shexp", "up_shexp", "down_shexp"):
        layer[k] = np.zeros_like(layer[k])  # the oracle always has a shared expert: with scales of 0 it adds nothing
    on_gpu = dict(layer, gate_shexp=None)
    gpu, off = MoELayer(on_gpu, max_tokens=50), MoELayer(on_gpu, max_tokens=50, no_tensor=True)
    for T in (9, 19, 20, 50):  # 90, 190, 200 and 500 assignments over 512 experts
        x = synth.make_input(T, 512, seed=T)
        # One code of an inner row of 256 values that rounds the other way moves an output by up to 6.5e-3 of the largest here
        # (its scale times the largest down weight and the expert's share, worked out in 64 bits): the layer's bar.
        out = check(layer, gpu, x, MAX_REL)
        groups = gpu.groups()
        assert groups[:, 2].max() == 2 and groups[:, 2].sum() == 10 * T  # every expert's rows are groups, none a tile
        assert np.array_equal(out, off.forward(x)) == by_integer_dots(gate, down, 10 * T), T
    gpu.close(), off.close()
