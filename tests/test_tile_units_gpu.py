"""On a B200: the tile kernels' decoders, which take a weight row in units of two stages, at row lengths that the decode
groups do not divide (a row's last half round) and at the shortest, against the CPU oracle."""
import pytest

from c0ven_b200 import MoELayer, synth
from test_gpu_parity import MAX_REL, TYPES, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("n_embd,n_ff", [(256, 256), (768, 1280), (1280, 768)])
def test_rows_that_end_in_half_a_round(t, n_embd, n_ff):
    layer = synth.make_layer(n_embd=n_embd, n_ff=n_ff, n_experts=32, n_used=4, gate_type=t, seed=t + n_embd)
    gpu = MoELayer(layer, max_tokens=400, tensor_min_rows=1)
    for T in (1, 17, 400):  # one tile of one row; an expert's rows in tiles of every length; several tiles in a row a CTA
        # 256 values a row: the weights' rounding to f16 alone, worked out in 64 bits, puts the worst element of Q6_K's 400 rows
        # at 1.063e-2 (longer rows average it out: 6.2e-3 at most here).
        check(layer, gpu, synth.make_input(T, n_embd, seed=T), 1.5e-2 if n_ff == 256 else MAX_REL)
    assert gpu.stats()["last_tensor_rows"] >= 400 * 4
    gpu.close()
