"""On a B200: the int8 tensor-instruction kernel for experts of a few rows, against the CPU oracle: as groups (with a
threshold for the tile kernels that no expert reaches; its arithmetic is the integer-dot kernels' but for f32 order) and as
the short end of the tile list, with experts of more rows on the tile kernels in the same step; at the shortest rows and at
lengths nothing is specialised for."""
import numpy as np
import pytest

from c0ven_b200 import MoELayer, synth
from test_gpu_parity import INT_PATH_REL, TYPES, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("n_embd,n_ff", [(256, 256), (768, 1280), (2048, 512), (4352, 256)])
def test_groups(t, n_embd, n_ff):
    layer = synth.make_layer(n_embd=n_embd, n_ff=n_ff, n_experts=64, n_used=4, gate_type=t, seed=t + n_embd)
    gpu = MoELayer(layer, max_tokens=200, tensor_min_rows=256)
    for T in (9, 16, 17, 65, 200):  # groups of up to two; with more rows than experts, of up to eight
        check(layer, gpu, synth.make_input(T, n_embd, seed=T), INT_PATH_REL)
    gpu.close()


@pytest.mark.parametrize("gate,down", [(t, t) for t in TYPES] + [(synth.Q4_K, synth.Q6_K), (synth.IQ4_XS, synth.IQ4_NL)])
def test_short_tiles_beside_long_ones(gate, down):
    """Rows that repeat route alike: experts that only one of the rows chose get its repeats, up to and past the 8 rows of
    one instruction and the 16 that an entry holds in a step that hits fewer than 256 experts; longer ones take the tiles."""
    layer = synth.make_layer(n_embd=768, n_ff=512, n_experts=320, n_used=4, gate_type=gate, down_type=down, seed=gate * 50 + down)
    repeats = [1, 7, 8, 9, 16, 17, 24, 25, 32, 33, 300, 2, 32]
    x = np.repeat(synth.make_input(len(repeats), 768, seed=3), repeats, axis=0)
    gpu = MoELayer(layer, max_tokens=len(x))
    check(layer, gpu, x)
    cnt = np.bincount(gpu.route(len(x))[0].reshape(-1), minlength=320)
    assert {1, 7, 8, 9, 16, 17, 24, 25, 32, 33, 300} <= set(cnt.tolist()) and np.count_nonzero(cnt) < 256
    gpu.close()


@pytest.mark.parametrize("gate,down", [(t, t) for t in TYPES] + [(synth.Q4_K, synth.Q6_K), (synth.IQ4_XS, synth.IQ4_NL)])
def test_entries_of_up_to_32_rows(gate, down):
    """A step that hits 256 experts or more: those of up to 32 rows are entries of the kernel, in all four of its forms, and
    longer ones stay on the tile kernels. (Below 256 the cut is at 16 rows: test_short_tiles_beside_long_ones.)"""
    layer = synth.make_layer(n_embd=768, n_ff=512, n_experts=320, n_used=4, gate_type=gate, down_type=down, seed=gate * 51 + down)
    repeats = list(range(9, 33))
    x = synth.make_input(340 + len(repeats), 768, seed=3)
    x = np.concatenate([x[len(repeats):], np.repeat(x[:len(repeats)], repeats, axis=0)])
    gpu = MoELayer(layer, max_tokens=len(x))
    check(layer, gpu, x)
    cnt = np.bincount(gpu.route(len(x))[0].reshape(-1), minlength=320)
    assert np.count_nonzero(cnt) >= 256 and 1280 <= cnt.sum() <= 24 * 320
    for lo, hi in ((1, 8), (9, 16), (17, 24), (25, 32), (33, 256)):
        assert np.count_nonzero((cnt >= lo) & (cnt <= hi)) >= 8, (lo, hi)
    assert len(gpu.groups()) == 0
    gpu.close()


@pytest.mark.parametrize("t", TYPES)
def test_both_lists_in_one_step(t):
    """Steps of 64 to 1,279 assignments over up to 128 experts whose threshold the pack lowers to two rows: the experts with
    one row are groups, the others the tile list, short enough for the kernel to take it whole (in the same launch where
    groups of that size are its own) and, with rows that repeat, with an expert too long for that."""
    layer = synth.make_layer(n_embd=512, n_ff=256, n_experts=128, n_used=4, gate_type=t, seed=t)
    gpu = MoELayer(layer, max_tokens=60)
    base = synth.make_input(60, 512, seed=t)
    for T, repeats in ((32, 1), (40, 1), (44, 1), (50, 12)):  # 128 assignments: groups of up to two; more: of up to eight
        x = np.concatenate([np.repeat(base[:1], repeats, axis=0), base[1:T - repeats + 1]])
        check(layer, gpu, x)
        cnt = np.bincount(gpu.route(T)[0].reshape(-1), minlength=128)
        assert (cnt.max() <= 8) == (repeats == 1)
        groups = gpu.groups()
        assert len(groups) == np.count_nonzero(cnt == 1) > 0
        assert gpu.stats()["last_tensor_rows"] - T == cnt[cnt > 1].sum() > 0  # T: the shared expert's rows
    gpu.close()


@pytest.mark.parametrize("t", TYPES)
def test_one_list_or_the_other(t):
    """Steps of 64 to 1,279 assignments: all experts on the tile list (few experts) or all on the groups' list, with and
    without one that needs the tile kernels."""
    layer = synth.make_layer(n_embd=512, n_ff=256, n_experts=320, n_used=4, gate_type=t, seed=t)
    gpu = MoELayer(layer, max_tokens=300)
    base = synth.make_input(300, 512, seed=t)
    for T, repeats in ((16, 1), (17, 4), (32, 1), (33, 1), (200, 1), (120, 20), (200, 40)):
        check(layer, gpu, np.concatenate([np.repeat(base[:1], repeats, axis=0), base[1:T - repeats + 1]]))
    gpu.close()


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("n_embd,n_ff", [(512, 256), (2048, 512)])
def test_a_layer_kept_off_the_tensor_cores_keeps_its_integer_dots(t, n_embd, n_ff):
    """MOE_FLAG_NO_TENSOR: the integer-dot kernels sum a row in one order however many rows a group holds (up to two, four at
    a time, eight), so a row's output has the same bits whatever step it comes in."""
    layer = synth.make_layer(n_embd=n_embd, n_ff=n_ff, n_experts=32, n_used=2, gate_type=t, seed=t)
    gpu = MoELayer(layer, max_tokens=65, no_tensor=True)
    x = synth.make_input(65, n_embd, seed=t)
    few = check(layer, gpu, x[:16], INT_PATH_REL).copy()
    assert gpu.groups()[:, 2].max() == 2
    for T in (40, 65):
        assert np.array_equal(check(layer, gpu, x[:T], INT_PATH_REL)[:16], few), T
        assert gpu.groups()[:, 2].max() > 4
    gpu.close()


@pytest.mark.parametrize("t", TYPES)
def test_entries_whose_rows_leave_room_for_one_cta(t):
    """The longest rows the kernel takes, of which two CTAs' 32 do not fit an SM in any type: one CTA of sixteen warps takes
    gate and up, with entries of every count of row tiles; a down product of more items than CTAs, each of which then takes
    runs of several entries."""
    n_embd = 2560 if t == synth.Q6_K else 2816
    layer = synth.make_layer(n_embd=n_embd, n_ff=256, n_experts=288, n_used=4, gate_type=t, seed=t + 7)
    repeats = list(range(9, 33))
    x = synth.make_input(300 + len(repeats), n_embd, seed=5)
    x = np.concatenate([x[len(repeats):], np.repeat(x[:len(repeats)], repeats, axis=0)])
    gpu = MoELayer(layer, max_tokens=len(x))
    check(layer, gpu, x)
    cnt = np.bincount(gpu.route(len(x))[0].reshape(-1), minlength=288)
    assert np.count_nonzero(cnt) >= 256 and 1280 <= cnt.sum() <= 24 * 288  # below 256 hit no entry passes 16 rows
    for lo, hi in ((1, 8), (9, 16), (17, 24), (25, 32)):
        assert np.count_nonzero((cnt >= lo) & (cnt <= hi)) >= 4, (lo, hi)
    assert len(gpu.groups()) == 0
    gpu.close()
