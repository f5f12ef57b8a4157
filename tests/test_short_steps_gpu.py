"""On a B200: steps of a few rows against the CPU oracle and against the same layer stage by stage (a profiled layer takes
its steps that way). One or two rows run in three launches: the router with the quantisers; gate/up with the top-k in
every CTA; the down product with the combine. Up to eight rows and 64 assignments take five: the top-k with the lists and
the combine have their own. Around the edges of the rules: 2 and 8 rows, 64 assignments, 128 units a weight row; and
router rows of every length a layer may have."""
import numpy as np
import pytest

from c0ven_b200 import MoELayer, synth
from oracle import oracle as O
from test_gpu_parity import INT_PATH_REL, TYPES, check

pytestmark = pytest.mark.gpu


def compare(layer, rows, seed=0, shared=True):
    on_gpu = layer if shared else dict(layer, gate_shexp=None)
    short, staged = MoELayer(on_gpu, max_tokens=64, no_tensor=True), MoELayer(on_gpu, max_tokens=64, no_tensor=True, profile=True)
    for T in rows:
        x = synth.make_input(T, layer["n_embd"], seed=seed + T)
        out = check(layer, short, x, INT_PATH_REL).copy()
        check(layer, staged, x, INT_PATH_REL)
        assert np.array_equal(short.groups(), staged.groups()), T
        for inner in (False, True):
            (q, d, bs), (q2, d2, bs2) = short.quantized(T, inner=inner), staged.quantized(T, inner=inner)
            if not inner:
                assert np.array_equal(q, q2) and np.array_equal(d, d2)
            # Inner rows: sums whose last bit may differ, so now and then a code that rounds the other way.
            assert np.abs(q.astype(np.int32) - q2).max() <= 1 and np.mean(q != q2) <= 1e-2
            assert np.allclose(d, d2, rtol=1e-3)
            if bs is not None and len(bs):
                assert np.array_equal(bs.reshape(-1), q.reshape(-1, 16).astype(np.int32).sum(1).astype(np.int16).reshape(-1))
        assert np.array_equal(short.forward(x), out)  # seen before: recorded; and once more from the recording
        assert np.array_equal(short.forward(x), out)
    short.close(), staged.close()


@pytest.mark.parametrize("t", TYPES)
def test_every_type(t):
    layer = synth.make_layer(n_embd=512, n_ff=512, n_experts=32, n_used=4, gate_type=t, seed=t)
    compare(layer, (1, 2, 3, 5, 8, 9))


@pytest.mark.parametrize("t", TYPES)
def test_every_type_in_lengths_nothing_is_specialised_for(t):
    layer = synth.make_layer(n_embd=768, n_ff=1280, n_experts=32, n_used=7, gate_type=t, shexp_gate_type=synth.Q8_0, shexp_down_type=t, seed=t)
    compare(layer, (1, 4, 8))


@pytest.mark.parametrize("n_used,rows", [(1, (1, 8)), (8, (7, 8)), (9, (7, 8)), (16, (4, 5))])
def test_assignments_around_the_limit_with_shared_experts(n_used, rows):
    layer = synth.make_layer(n_embd=512, n_ff=256, n_experts=32, n_used=n_used, gate_type=synth.Q4_K, down_type=synth.Q6_K,
                             shexp_gate_type=synth.Q8_0, shexp_down_type=synth.Q8_0, zipf_s=1.1, seed=n_used)
    compare(layer, rows)


@pytest.mark.parametrize("n_ff", [2048, 2304, 4096])
def test_weight_rows_around_the_longest(n_ff):
    layer = synth.make_layer(n_embd=256, n_ff=n_ff, n_experts=32, n_used=4, gate_type=synth.Q4_K, down_type=synth.Q8_0, seed=n_ff)
    compare(layer, (1, 8))


def test_without_a_shared_expert_and_equal_logits():
    layer = synth.make_layer(n_embd=512, n_ff=256, n_experts=32, n_used=4, gate_type=synth.Q8_0, seed=33)
    for k in ("gate_shexp", "up_shexp", "down_shexp"):
        layer[k] = np.zeros_like(layer[k])  # the oracle always has one: with scales of 0 it adds nothing
    layer["router"][5] = layer["router"][2]
    compare(layer, (1, 3, 8), shared=False)
    gpu = MoELayer(dict(layer, gate_shexp=None), max_tokens=8)
    x = np.zeros((2, 512), dtype=np.float32)
    assert np.all(gpu.forward(x) == 0)
    assert np.array_equal(gpu.route(2)[0], O.moe_forward(layer, x)[1])
    gpu.close()


@pytest.mark.parametrize("n_embd,no_tensor", [(8192, False), (8192, True), (16384, False), (16384, True)])
def test_the_router_on_the_longest_rows(n_embd, no_tensor):
    """Rows of up to 16,384 values: the kernel of one row holds all of it in shared memory, the others a ring of stages whatever
    the length; and the longer steps of a layer kept off the tensor cores, in several CTAs' worth of rows."""
    layer = synth.make_layer(n_embd=n_embd, n_ff=256, n_experts=32, n_used=2, gate_type=synth.Q4_K, down_type=synth.Q8_0, seed=n_embd)
    gpu = MoELayer(layer, max_tokens=70, no_tensor=no_tensor)
    for T in (1, 2, 9, 64, 70):
        check(layer, gpu, synth.make_input(T, n_embd, seed=T))
    gpu.close()


def test_layers_of_several_row_lengths_in_turn():
    """The router's kernels are shared by the process's layers: a layer of shorter rows leaves those of longer ones running."""
    layers = [synth.make_layer(n_embd=n, n_ff=256, n_experts=32, n_used=2, gate_type=synth.Q8_0, seed=n) for n in (7168, 2048, 512)]
    gpus = [MoELayer(layer, max_tokens=70, no_tensor=True) for layer in layers]
    for T in (70, 2):
        for layer, gpu in list(zip(layers, gpus)) + [(layers[0], gpus[0])]:
            check(layer, gpu, synth.make_input(T, layer["n_embd"], seed=T))
    for gpu in gpus:
        gpu.close()


@pytest.mark.parametrize("n_embd,n_experts", [(256, 32), (768, 96), (2304, 512)])
def test_exact_router_at_the_edges_of_its_forms(n_embd, n_experts):
    """One row, 8 and 32 rows a CTA and one more than each, the longest step; rows of one stage's length a piece and of lengths
    whose stages the ring does not divide; the oracle's ids bit for bit (check)."""
    layer = synth.make_layer(n_embd=n_embd, n_ff=256, n_experts=n_experts, n_used=4, gate_type=synth.Q8_0, seed=n_embd)
    gpu = MoELayer(layer, max_tokens=64)
    for T in (1, 2, 8, 9, 32, 33, 64):
        check(layer, gpu, synth.make_input(T, n_embd, seed=T))
    gpu.close()
