"""What the MoE expert layer is timed on: one pass of a layer over a step's rows, as an engine's step loop makes it.

A case says the layer (sizes, weight types, skew of its routing), the rows of the step and the way in:

- "device": `MoELayer.forward_device`, rows resident in device memory (a decode, draft-verify or prefill step);
- "stack": `rmsnorm_rows_device` and `MoELayer.forward_residual_device` over two layers, x <- x + moe(norm(x));
- "host": `MoELayer.forward`, page-locked host rows in and out, with the chunks the benchmark uses.

Weights are random blocks with the value distributions of `c0ven_b200.synth`, made on the GPU because a layer's are up to
1.7 GB; rows are N(0, 1). Everything comes from the seed.
"""
import numpy as np
import torch

from c0ven_b200 import MoELayer, synth
from c0ven_b200.layer import rmsnorm_rows_device

# Sizes: "full" is the benchmark's layer; "wide" has sizes that no kernel is specialised for, and no shared expert;
# "small" is a smaller model's layer.
SHAPES = {"full": dict(n_embd=2048, n_ff=512, n_experts=512, n_used=10, shared=True),
          "wide": dict(n_embd=2560, n_ff=768, n_experts=128, n_used=8, shared=False),
          "small": dict(n_embd=1024, n_ff=512, n_experts=64, n_used=4, shared=True)}

# Weight types that go together in a file: gate and up, down, the shared expert's gate and up, its down. The i-quant
# pairs are the ones the reference's model uses (gate and up in one, down in IQ4_NL or Q2_0, the shared expert Q8_0).
TYPES = {"q8_0": ("Q8_0", "Q8_0", "Q8_0", "Q8_0"),
         "q4_k": ("Q4_K", "Q4_K", "Q4_K", "Q4_K"),
         "q4_k_mix": ("Q4_K", "Q6_K", "Q8_0", "Q8_0"),
         "iq3_s": ("IQ3_S", "IQ3_S", "IQ3_S", "IQ3_S"),
         "iq4_xs_nl": ("IQ4_XS", "IQ4_NL", "Q8_0", "Q8_0"),
         "iq3_xxs_nl": ("IQ3_XXS", "IQ4_NL", "Q8_0", "Q8_0"),
         "iq2_s_q2": ("IQ2_S", "Q2_0", "Q8_0", "Q8_0")}

# The f16 scales of a block: (byte offset, lowest, highest), as synth.random_blocks draws them.
SCALES = {"Q8_0": [(0, 1e-4, 3e-4)], "Q4_K": [(0, 1e-4, 1e-3), (2, 1e-4, 1e-3)], "Q6_K": [(208, 2e-5, 2e-4)],
          "IQ3_S": [(0, 1e-4, 1e-3)], "IQ3_XXS": [(0, 1e-4, 1e-3)], "IQ2_S": [(0, 2.5e-4, 2.5e-3)],
          "Q2_0": [(0, 5e-3, 2e-2)], "IQ4_NL": [(0, 1e-4, 3e-4)], "IQ4_XS": [(0, 5e-6, 2e-5)]}


def listed():
    case = lambda name, way, shape, types, tokens, zipf: dict(name=name, way=way, shape=shape, types=types, tokens=tokens, zipf=zipf)  # noqa: E731
    return [
        # One token of one request: the decode step, bound by launches and by reading ten experts once.
        case("decode1_q8_0", "device", "full", "q8_0", 1, 0.0),
        # A few requests decoding together, mixed types, skewed routing: some experts shared by rows.
        case("decode4_q4_k_mix_zipf", "device", "full", "q4_k_mix", 4, 1.1),
        # Draft-verify of a couple of requests in the smallest types, on a layer of sizes nothing is specialised for.
        case("verify13_iq2_s_wide", "device", "wide", "iq2_s_q2", 13, 0.0),
        # Four requests of eight drafted rows through consecutive layers, as a stack runs them.
        case("stack32_iq3_s", "stack", "full", "iq3_s", 32, 0.0),
        # A busy server's decode batch: about two rows an expert over every expert, the largest weights.
        case("batch100_q8_0", "device", "full", "q8_0", 100, 0.0),
        # A short prompt chunk or a large decode batch with skewed routing.
        case("batch256_q4_k_mix_zipf", "device", "full", "q4_k_mix", 256, 1.1),
        # A prompt of odd length, even routing: about fifteen rows an expert.
        case("prompt777_q4_k", "device", "full", "q4_k", 777, 0.0),
        # A packed ragged batch of runs 1, 8, 512 and 3000 with skewed routing (the benchmark's second configuration).
        case("ragged3521_q4_k_zipf", "device", "full", "q4_k", 3521, 1.1),
        # The same kind of batch by the host-buffer call, copies included, in IQ3_XXS and IQ4_NL.
        case("host1500_iq3_xxs_nl", "host", "full", "iq3_xxs_nl", 1500, 1.1),
        # The reference's prompt chunk.
        case("prompt4352_iq4_xs_nl", "device", "full", "iq4_xs_nl", 4352, 0.0),
        # The largest step of the benchmark's sweep.
        case("sweep8192_q4_k_mix_zipf", "device", "full", "q4_k_mix", 8192, 1.1),
        # A long prompt in one step: the benchmark's headline.
        case("prefill32768_q4_k", "device", "full", "q4_k", 32768, 0.0),
    ]


def draw(rng):
    shape = rng.choice(["full", "full", "full", "wide", "small"])
    way = rng.choice(["device"] * 6 + ["stack", "host"])
    most = {"device": 16384, "stack": 1024, "host": 4096}[way]
    tokens = int(round(most ** rng.random()))
    return dict(way=way, shape=shape, types=rng.choice(sorted(TYPES)), tokens=max(1, tokens), zipf=rng.choice([0.0, 0.0, 1.1]))


def _blocks(name, rows, cols, gen):
    """rows x cols random weights as the file's blocks, uint8 [rows, row bytes] on the host."""
    t = synth.TYPE_IDS[name]
    n = rows * cols // synth.BLOCK_VALUES[t]
    b = torch.randint(0, 256, (n, synth.BLOCK_BYTES[t]), dtype=torch.uint8, device="cuda", generator=gen)
    if name == "Q8_0":  # codes in -127 .. 127
        b[b == 128] = 129
    for at, lo, hi in SCALES[name]:
        d = torch.rand((n, 1), device="cuda", generator=gen) * (hi - lo) + lo
        b[:, at:at + 2] = d.half().view(torch.uint8)
    return b.cpu().numpy().reshape(rows, synth.row_bytes(t, cols))


def _layer(case, seed):
    s = SHAPES[case["shape"]]
    E, F, NE, K = s["n_embd"], s["n_ff"], s["n_experts"], s["n_used"]
    gate, down, sgate, sdown = TYPES[case["types"]]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    L = dict(n_embd=E, n_ff=F, n_experts=NE, n_used=K, gate_type=synth.TYPE_IDS[gate], down_type=synth.TYPE_IDS[down],
             shexp_gate_type=synth.TYPE_IDS[sgate], shexp_down_type=synth.TYPE_IDS[sdown])
    L["router"] = (torch.randn((NE, E), device="cuda", generator=gen) * 0.02).cpu().numpy()
    L["router_bias"] = synth.zipf_bias(NE, case["zipf"], rng) if case["zipf"] else None
    L["gate_exps"] = _blocks(gate, NE * F, E, gen).reshape(NE, F, -1)
    L["up_exps"] = _blocks(gate, NE * F, E, gen).reshape(NE, F, -1)
    L["down_exps"] = _blocks(down, NE * E, F, gen).reshape(NE, E, -1)
    if s["shared"]:
        L["shexp_gate_inp"] = (torch.randn(E, device="cuda", generator=gen) * 0.02).cpu().numpy()
        L["gate_shexp"], L["up_shexp"] = _blocks(sgate, F, E, gen), _blocks(sgate, F, E, gen)
        L["down_shexp"] = _blocks(sdown, E, F, gen)
    return L


def _chunk_rows(tokens):
    """Rows a chunk of a host-buffer call takes, as the benchmark sets it."""
    return 8192 if tokens >= 16384 else tokens // 2 if tokens >= 2048 else 0


_stream = None


def stream():
    """The program's compute stream: every layer's calls are queued on it."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def prepare(case, seed):
    T, E = case["tokens"], SHAPES[case["shape"]]["n_embd"]
    nlayers = 2 if case["way"] == "stack" else 1
    layers = [MoELayer(_layer(case, seed * 2 + i), max_tokens=T, host_chunk_rows=_chunk_rows(T) if case["way"] == "host" else 0) for i in range(nlayers)]
    x = torch.randn((T, E), device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed + 7919))
    state = dict(way=case["way"], layers=layers, x=x, T=T, E=E)
    if case["way"] == "host":
        state["x"] = x.cpu().pin_memory()
        state["out"] = torch.empty((T, E), dtype=torch.float32).pin_memory()
    else:
        state["out"] = torch.empty_like(x)
        state["norm"] = torch.empty_like(x) if case["way"] == "stack" else None
    torch.cuda.synchronize()
    return state


def run(state):
    layers, T, x, out = state["layers"], state["T"], state["x"], state["out"]
    if state["way"] == "host":
        layers[0].forward(x.numpy(), out.numpy())
    elif state["way"] == "device":
        layers[0].forward_device(x.data_ptr(), T, out.data_ptr(), stream().cuda_stream)
    else:
        st, norm = stream().cuda_stream, state["norm"]
        for layer in layers:
            rmsnorm_rows_device(x.data_ptr(), None, T, state["E"], 1e-6, norm.data_ptr(), st)
            layer.forward_residual_device(norm.data_ptr(), T, x.data_ptr(), out.data_ptr(), st)
            x = out
    return out


def _experts_hit(case):
    """Distinct experts a step hits: exact in expectation for even routing, else by routing sampled logits with the bias."""
    s = SHAPES[case["shape"]]
    NE, K, T = s["n_experts"], s["n_used"], case["tokens"]
    if not case["zipf"]:
        return NE * (1.0 - (1.0 - K / NE) ** T)
    rng = np.random.default_rng(1)
    bias = synth.zipf_bias(NE, case["zipf"], rng)
    logits = rng.standard_normal((min(T, 4096), NE)).astype(np.float32) * (0.02 * s["n_embd"] ** 0.5) + bias
    return float(len(np.unique(np.argpartition(-logits, K - 1, axis=1)[:, :K])))


def work(case):
    s = SHAPES[case["shape"]]
    E, F, NE, K, T = s["n_embd"], s["n_ff"], s["n_experts"], s["n_used"], case["tokens"]
    gate, down, sgate, sdown = (synth.TYPE_IDS[t] for t in TYPES[case["types"]])
    n = 2 if case["way"] == "stack" else 1
    weights = (NE + s["shared"]) * E * 4 + _experts_hit(case) * synth.expert_bytes(gate, down, E, F)
    flops = 2 * E * (NE + s["shared"]) + K * 6 * E * F
    if s["shared"]:
        weights += synth.expert_bytes(sgate, sdown, E, F)
        flops += 6 * E * F
    return {"bytes": n * weights + 2 * T * E * 4, "flops": float(n * T * flops)}


def tolerance(case):
    # Four times what the integer-dot kernels and the tensor-core kernels were measured to differ by on the same steps (3
    # and 300 rows, every type, two shapes): the same quantised rows, f32 sums in another order or f16 products, and now
    # and then a code of an inner row that rounds the other way. Q4_K throughout: rel 5e-4, max 2e-3 (more over more
    # values); the other types, whose weights keep more bits than f16 products do: rel 4e-3, max 7e-2.
    return {"rel": 2e-3, "max": 0.03} if case["types"] == "q4_k" else {"rel": 1.5e-2, "max": 0.25}
