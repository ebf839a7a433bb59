"""The calls whose time is measured: what users of this library have it do, through its public entry points.

Each case is one attention call (or one step of a sampling run) on tensors that a program already holds on the GPU.  The families:

``self``       ``int8_attention`` without a mask on head-major Q/K/V of one length: a transformer's self-attention
``cross``      the same with a query and a key length of their own, on token-major tensors (views of ``[B, N, H*D]``)
``causal``     self-attention of a prefill under the causal rule
``bias``       an additive mask of its own for every query (FP32 or BF16)
``rows``       a boolean mask per query in which some queries see nothing; operands packed first, LSE wanted (window merging)
``keys``       a batch of sequences of different lengths, padded: one boolean mask per sequence
``gather``     keys re-ordered by a validated permutation, read through the table
``construct``  dense attention that also freezes the retained-mass pattern (the first step of a sampling run)
``reuse``      attention over the tiles of a frozen pattern, on inputs that have drifted since (the later steps)
"""
import math

import torch

import risaattention_b200 as risa

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
THETA = 0.99          # retained mass of every pattern
CLUSTERS = 2          # token groups of the sparse workloads: about half of the key tiles are kept
EMPTY_ROWS = 0.1      # share of queries that a "rows" mask hides everything from
DEFAULTS = {"batch": 1, "head_dim": 128, "dtype": "bf16", "v": "absmax", "lse": False}


def _case(family, q_heads, kv_heads, q_len, k_len=None, name=None, **more):
    case = {"family": family, "q_heads": q_heads, "kv_heads": kv_heads, "q_len": q_len,
            "k_len": q_len if k_len is None else k_len, **DEFAULTS, **more}
    return case if name is None else {"name": name, **case}


def listed():
    return [
        # The shortest sequence of the dense sweep: a call whose time is launches and host work.
        _case("self", 16, 4, 512, name="self_512"),
        # FP32 operands with LSE at the length up to which 64-key tiles are used: small windows that are merged afterwards.
        _case("self", 16, 4, 1024, dtype="f32", lse=True, name="self_1k_f32_lse"),
        # The ordinary image-model length, with the centred value quantisation.
        _case("self", 16, 4, 2048, v="midpoint_affine", name="self_2k_affine"),
        # The headline call: one long sequence, four query heads to a key/value head.
        _case("self", 16, 4, 32768, name="self_32k"),
        # Text conditioning of a video model: many queries, a short ragged key sequence, token-major storage.
        _case("cross", 24, 24, 7800, 333, name="cross_7800x333"),
        # Heads of 256 channels over a key sequence four times the query's.
        _case("self", 32, 8, 4096, 16384, head_dim=256, name="wide_4kx16k_d256"),
        # A language model's prefill: causal, 64 channels, half precision.
        _case("causal", 32, 8, 4096, head_dim=64, dtype="f16", name="causal_4k_d64"),
        # A learned or relative-position bias of every (head, query, key).
        _case("bias", 32, 8, 4096, head_dim=64, dtype="bf16", mask="f32", name="bias_4k_d64"),
        # A window of visible keys per query, quantised once and attended with LSE.
        _case("rows", 16, 4, 2048, batch=2, lse=True, name="rows_2k_b2_lse"),
        # A padded batch of sequences of ragged length, 80-channel heads.
        _case("keys", 16, 16, 1500, batch=4, head_dim=80, dtype="f16", name="keys_1500_b4_d80"),
        # The first step of a sampling run: dense output and the pattern it freezes.
        _case("construct", 16, 4, 8192, name="construct_8k"),
        # A later step of a video model's run: all 40 heads, 21 x 30 x 52 tokens, through the frozen pattern.
        _case("reuse", 40, 40, 32760, name="reuse_video_32760"),
    ]


def draw(rng):
    largest = max(work(c)["flops"] for c in listed())
    most_mask = 32 * 4096 * 4096  # entries of the largest listed mask

    def length(low, high):
        n = round(math.exp(rng.uniform(math.log(low), math.log(high))))
        return max(low, n - n % 128 if rng.random() < 0.4 else n)

    while True:
        family = rng.choice(("self", "self", "self", "cross", "causal", "bias", "rows", "keys", "gather", "construct", "reuse"))
        q_heads, kv_heads = rng.choice(((16, 4), (16, 16), (32, 8), (24, 24), (40, 40), (8, 1)))
        case = _case(family, q_heads, kv_heads, 0, batch=rng.choice((1, 1, 1, 2, 4)), dtype=rng.choice(("bf16", "bf16", "bf16", "f16", "f32")),
                     head_dim=rng.choice((64, 80, 128, 128, 128, 256)), v=rng.choice(("absmax", "absmax", "midpoint_affine")))
        if family == "self":
            case["q_len"] = case["k_len"] = length(128, 32768)
            case["lse"] = rng.random() < 0.25
        elif family == "cross":
            case["q_len"], case["k_len"] = length(256, 32768), length(77, 4096)
        elif family in ("causal", "gather"):
            case["q_len"] = case["k_len"] = length(256, 16384)
        elif family in ("bias", "rows", "keys"):
            case["q_len"] = case["k_len"] = length(256, 4096)
            if family == "bias":
                case["mask"] = rng.choice(("f32", "bf16"))
            case["lse"] = family == "rows"
        else:
            case.update(batch=1, head_dim=128, dtype="bf16", q_len=length(4096, 32768))
            case["k_len"] = case["q_len"]
        entries = case["batch"] * q_heads * case["q_len"] * case["k_len"] if family in ("bias", "rows") else 0
        if work(case)["flops"] <= largest and entries <= most_mask:
            return case


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, dtype, *shape):
    return torch.randn(*shape, device="cuda", generator=g).to(dtype)


def _clustered(case, g):
    """N(0, 1) Q and K to which each 128-token block adds one of the head's prototypes of norm 8, and N(0, 1) V."""
    q_heads, kv_heads, n, d = case["q_heads"], case["kv_heads"], case["q_len"], case["head_dim"]
    q, k, v = (_normal(g, torch.bfloat16, 1, h, n, d) for h in (q_heads, kv_heads, kv_heads))
    prototypes = torch.randn(1, kv_heads, CLUSTERS, d, device="cuda", generator=g)
    prototypes *= 8.0 / prototypes.norm(dim=-1, keepdim=True)
    prototypes = prototypes.bfloat16()
    cluster = torch.arange(n, device="cuda").div(128, rounding_mode="floor") % CLUSTERS
    q += prototypes.repeat_interleave(q_heads // kv_heads, dim=1)[:, :, cluster]
    k += prototypes[:, :, cluster]
    return q, k, v


def _mask(case, g):
    batch, heads, n, k_len = case["batch"], case["q_heads"], case["q_len"], case["k_len"]
    if case["family"] == "bias":
        return torch.randn(batch, heads, n, k_len, device="cuda", generator=g, dtype=DTYPES[case["mask"]])
    if case["family"] == "rows":
        mask = torch.rand(batch, heads, n, k_len, device="cuda", generator=g) < 0.9
        mask[:, :, torch.randperm(n, device="cuda", generator=g)[: int(n * EMPTY_ROWS)]] = False
        return mask
    # lengths spread evenly from half the padded length to all of it, in random order
    lengths = torch.linspace(0.5, 1.0, batch + 1, device="cuda")[1:] * k_len
    lengths = lengths.round().long()[torch.randperm(batch, device="cuda", generator=g)]
    return (torch.arange(k_len, device="cuda") < lengths[:, None])[:, None, None, :]


def prepare(case, seed):
    g = _generator(seed)
    dtype, batch, d = DTYPES[case["dtype"]], case["batch"], case["head_dim"]
    state = {"case": case, "options": {"v_quantization": case["v"]}}
    if case["family"] in ("construct", "reuse"):
        q, k, v = _clustered(case, g)
        if case["family"] == "reuse":
            _, state["pattern"] = risa.construct_sparse_int8_attention(q, k, v, theta=THETA, **state["options"])
            for x in (q, k, v):  # a later step of the run
                x += 0.05 * _normal(g, torch.bfloat16, *x.shape)
    else:
        sizes = ((case["q_heads"], case["q_len"]), (case["kv_heads"], case["k_len"]), (case["kv_heads"], case["k_len"]))
        if case["family"] == "cross":
            q, k, v = (_normal(g, dtype, batch, n, h * d).view(batch, n, h, d).transpose(1, 2) for h, n in sizes)
        else:
            q, k, v = (_normal(g, dtype, batch, h, n, d) for h, n in sizes)
    if case["family"] in ("bias", "rows", "keys"):
        state["options"]["attn_mask"] = _mask(case, g)
    if case["family"] == "causal":
        state["options"]["is_causal"] = True
    if case["family"] == "gather":
        order = torch.rand(batch, case["kv_heads"], case["k_len"], device="cuda", generator=g).argsort(dim=-1)
        state["options"]["kv_permutation"] = risa.prepare_kv_permutation(order)
    return dict(state, q=q, k=k, v=v)


def run(state):
    family, lse = state["case"]["family"], state["case"]["lse"]
    q, k, v, options = state["q"], state["k"], state["v"], state["options"]
    if family == "construct":
        out, pattern = risa.construct_sparse_int8_attention(q, k, v, theta=THETA, **options)
        # the ids of the kept tiles in a buffer of one size, so that the patterns of different inputs can be held side by side
        tiles = pattern.block_indices.numel() / pattern.coverage
        ids = torch.nn.functional.pad(pattern.block_indices, (0, round(tiles) - pattern.block_indices.numel()))
        return out, pattern.row_offsets, ids, pattern.measured_retained_mass
    if family == "reuse":
        return risa.sparse_int8_attention(q, k, v, state["pattern"], output_layout="nhd", **options)
    if family == "rows":
        packed = risa.prequantize_int8_attention(q, k, v, return_lse=True, **options)
        return risa.int8_attention_from_prequantized(packed, return_lse=True)
    return risa.int8_attention(q, k, v, return_lse=lse, **options)


def work(case):
    """Q, K, V and the mask read once, output (and LSE) written once; two multiply-adds per visible (query, key, channel)."""
    size = 4 if case["dtype"] == "f32" else 2
    batch, q_heads, kv_heads, d = case["batch"], case["q_heads"], case["kv_heads"], case["head_dim"]
    queries, keys = batch * q_heads * case["q_len"], batch * kv_heads * case["k_len"]
    pairs = queries * case["k_len"]
    moved = size * d * (2 * queries + 2 * keys) + (4 * queries if case["lse"] else 0)
    family = case["family"]
    if family == "causal":
        pairs = queries * (case["q_len"] + 1) / 2
    elif family == "bias":
        moved += pairs * (4 if case["mask"] == "f32" else 2)
    elif family == "rows":
        moved += pairs
        pairs *= 1 - EMPTY_ROWS
    elif family == "keys":
        moved += batch * case["k_len"]
        pairs *= (1.5 + 0.5 / batch) / 2  # the mean of the lengths
    elif family == "gather":
        moved += 4 * keys
    elif family == "reuse":
        pairs /= CLUSTERS
    return {"bytes": moved, "flops": 4 * pairs * d}


def tolerance(case):
    # Outputs are rounded to the 16-bit input type (bf16 for FP32 operands): half a unit in the last place on each side,
    # and single steps of the 8-bit probabilities where two exponentials round differently.
    if case["dtype"] == "f16":
        return {"rel": 2e-3, "max": 1e-2}
    return {"rel": 5e-3, "max": 2e-2}
