"""Kernels at the edges of their ranges: remainders of tiles, the smallest and the largest sizes a branch of
a dispatch takes, against the CPU oracle or the tensor program a kernel replaces."""

import numpy as np
import pytest
import torch

from oracle import c_oracle
from sage_b200 import sage_dequantize, synthetic_sage
from sage_b200.packing import direction_codebook_from_logits, pack_spherical, pack_spherical_radii

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [128, 2560, 5120, 11264, 11392, 25600])
@pytest.mark.parametrize("n", [1, 17])
@pytest.mark.parametrize("offset", [0, 1])
def test_dense_dequantisation_blocks_and_windows(k, n, offset):
    """Rows that do not fill a block of eight, one to three windows of channels, both block sizes, and a
    permutation that is not 16-byte aligned."""
    cpu = synthetic_sage(k, n, seed=k + n)
    gpu = {key: value.cuda() for key, value in cpu.items()}
    if offset:
        gpu["permutation"] = torch.cat([gpu["permutation"][:1], gpu["permutation"]])[1:]
    weight = sage_dequantize(gpu["packed_codes"], gpu["radius_codes"], gpu["radius_grid"], gpu["codebook"],
                             gpu["permutation"], n)
    assert np.array_equal(weight.cpu().numpy().view(np.uint16), c_oracle.decode_fp16(cpu, n).view(np.uint16))


@pytest.mark.parametrize("entries", [64, 128, 256])
@pytest.mark.parametrize("n,k", [(1, 128), (19, 384), (33, 2560)])
@pytest.mark.parametrize("index", [torch.int32, torch.int64, torch.int16])
def test_packing_from_logits(entries, n, k, index):
    """The one-pass packing of a checkpoint's logits equals softplus, the radii's packing and the codebook's
    tensor program bit for bit; an identity permutation comes back empty."""
    gen = torch.Generator().manual_seed(entries + n)
    state = {
        "signs": (torch.randint(0, 2, (n, k), generator=gen, dtype=torch.int8) * 2 - 1).cuda(),
        "direction_indices": torch.randint(0, entries, (n, k // 8), generator=gen).to(index).cuda(),
        "radius_logits": (torch.randn(n, k // 8, generator=gen) * 12).cuda(),
        "angle_logits": (torch.randn(entries, 7, generator=gen) * 3).cuda(),
        "radius_bits": torch.tensor(10 - (entries.bit_length() - 1)), "group_size": torch.tensor(128),
        "sage_version": torch.tensor(1),
    }
    want = pack_spherical_radii(state["signs"], state["direction_indices"],
                                torch.nn.functional.softplus(state["radius_logits"]), entries, sage=True)
    book = direction_codebook_from_logits(state["angle_logits"]).half().reshape(entries, 4, 2).permute(1, 0, 2)
    for order in (torch.randperm(k, generator=gen), torch.arange(k)):
        state["channel_unpermutation"] = order.cuda()
        got = pack_spherical(state, sage=True)
        for key in want:
            assert torch.equal(got[key], want[key]), key
        assert torch.equal(got["codebook"], book)
        identity = bool((order == torch.arange(k)).all())
        assert torch.equal(got["permutation"].cpu(), torch.empty(0, dtype=torch.int32) if identity else order.argsort().int())


@pytest.mark.parametrize("hidden,inter,experts", [(512, 128, 40), (2048, 768, 36), (256, 1152, 33)])
@pytest.mark.parametrize("rows", [1, 8, 9, 16])
def test_expert_mlp_blocks(hidden, inter, experts, rows):
    """Blocks of the routed-expert kernels: one and two operand blocks of rows, a partial item of weight tiles, few
    groups of K, unused blocks and foreign experts (zeros), against FP32 matmuls on the dense weights."""
    from sage_b200.experts import SAGEExperts, expert_slice, synthetic_expert_stack

    first = 5
    stacks = [synthetic_expert_stack(k, n, experts, 21 + j, "cuda", direction_bits=6 + j, first=first)
              for j, (k, n) in enumerate(((hidden, inter), (hidden, inter), (inter, hidden)))]
    module = SAGEExperts(*stacks, first_expert=first)
    gen = torch.Generator(device="cuda").manual_seed(hidden + rows)
    x = torch.randn(experts, rows, hidden, generator=gen, device="cuda").half()
    ids = torch.arange(experts, dtype=torch.int32, device="cuda") + first
    ids[3], ids[7] = -1, first + experts
    got = module.forward_blocks(x, ids).float()

    def dense(stack, expert, n):
        one = expert_slice(stack, expert)
        return sage_dequantize(*[one[key] for key in ("packed_codes", "radius_codes", "radius_grid", "codebook",
                                                      "permutation")], n).float()

    for b in (0, 3, 7, 8, experts - 1):
        if b in (3, 7):
            assert not got[b].any()
            continue
        gate, up = x[b].float() @ dense(stacks[0], b, inter).T, x[b].float() @ dense(stacks[1], b, inter).T
        want = (torch.nn.functional.silu(gate) * up).half().float() @ dense(stacks[2], b, hidden).T
        assert ((got[b] - want).norm(dim=-1) / want.norm(dim=-1)).max() < 2e-3


@pytest.mark.parametrize("hidden,inter", [(3328, 256), (256, 3328), (2176, 2048)])
@pytest.mark.parametrize("rows", [8, 16])
def test_expert_mlp_beyond_a_vector_per_thread(hidden, inter, rows):
    """More than 2048 channels, up to the most that fit beside 64 entries with two operand blocks: threads come to
    several vectors, and to another operand block's, of one permutation."""
    from sage_b200 import _lib
    from sage_b200.experts import SAGEExperts, expert_slice, synthetic_expert_stack

    assert _lib.load().sageb200_expert_mlp_fits(rows, hidden, inter, 64) == 1
    assert _lib.load().sageb200_expert_mlp_fits(16, 3456, 128, 64) == 0
    experts = 33
    stacks = [synthetic_expert_stack(k, n, experts, 31 + j, "cuda", direction_bits=6)
              for j, (k, n) in enumerate(((hidden, inter), (hidden, inter), (inter, hidden)))]
    module = SAGEExperts(*stacks)
    x = torch.randn(experts, rows, hidden, generator=torch.Generator(device="cuda").manual_seed(rows), device="cuda").half()
    got = module.forward_blocks(x, torch.arange(experts, dtype=torch.int32, device="cuda")).float()
    names = ("packed_codes", "radius_codes", "radius_grid", "codebook", "permutation")
    for b in (0, experts - 1):
        gate, up, down = (sage_dequantize(*[expert_slice(stack, b)[key] for key in names], n).float()
                          for stack, n in zip(stacks, (inter, inter, hidden)))
        want = (torch.nn.functional.silu(x[b].float() @ gate.T) * (x[b].float() @ up.T)).half().float() @ down.T
        assert ((got[b] - want).norm(dim=-1) / want.norm(dim=-1)).max() < 2e-3


@pytest.mark.parametrize("rows", [512, 515, 1026])
@pytest.mark.parametrize("hidden", [128, 2560])
def test_permuting_passes_of_four_rows(rows, hidden):
    """Norm, SwiGLU and gather of many rows, four at a time, with a shorter last block: bit for bit the one-row
    kernels and an index_select."""
    import ctypes

    from sage_b200 import SAGELinear, _lib

    lib, vp = _lib.load(), lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else None)  # noqa: E731
    gen = torch.Generator(device="cuda").manual_seed(rows)
    draw = lambda *shape: torch.randn(*shape, generator=gen, device="cuda").half()  # noqa: E731
    perms = [torch.randperm(hidden, generator=gen, device="cuda").int() for _ in range(3)]
    residual, delta, weight = draw(rows, hidden), draw(rows, hidden), draw(hidden)
    for d in (delta, None):
        plain, four, x, outs = residual.clone(), residual.clone(), torch.empty_like(residual), [torch.empty_like(residual) for _ in perms]
        assert lib.sageb200_glue_add_rmsnorm(vp(plain), vp(d), vp(weight), vp(x), rows, hidden, 1e-6, None) == 0
        array = ctypes.c_void_p * 3
        assert lib.sageb200_glue_add_rmsnorm_permuted(vp(four), vp(d), vp(weight), None, array(*[p.data_ptr() for p in perms]),
                                                      array(*[o.data_ptr() for o in outs]), 3, rows, hidden, 1e-6, None) == 0
        assert torch.equal(plain, four)
        for perm, out in zip(perms, outs):
            assert torch.equal(out, x[:, perm.long()])
    gate, up, act, got = draw(rows, hidden), draw(rows, hidden), torch.empty_like(residual), torch.empty_like(residual)
    assert lib.sageb200_glue_swiglu(vp(gate), vp(up), vp(act), act.numel(), None) == 0
    assert lib.sageb200_glue_swiglu_permuted(vp(gate), vp(up), vp(perms[0]), vp(got), rows, hidden, 148, None) == 0
    assert torch.equal(got, act[:, perms[0].long()])
    packed = {key: value.cuda() for key, value in synthetic_sage(hidden, 48, seed=1).items()}
    plain = dict(packed, permutation=packed["permutation"][:0])
    assert torch.equal(SAGELinear(packed, 48)(gate), SAGELinear(plain, 48)(gate[:, packed["permutation"].long()].contiguous()))


@pytest.mark.parametrize("rows,k,n", [(17, 2560, 1024), (33, 256, 129), (16, 9728, 2560), (300, 640, 1025), (600, 1280, 256)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("permuted", [False, True])
def test_linear_in_a_typed_model(rows, k, n, dtype, permuted):
    """BF16 or FP16 rows with and without a bias through one GEMM launch: bit for bit the FP16 operator with the
    conversions and the addition as separate operations (a bias of another type takes those)."""
    from sage_b200 import SAGELinear, sage

    packed = {key: value.cuda() for key, value in synthetic_sage(k, n, seed=rows, permuted=permuted).items()}
    gen = torch.Generator(device="cuda").manual_seed(rows + n)
    x = torch.randn(rows, k, generator=gen, device="cuda").to(dtype)
    plain = sage(x.half(), *[packed[key] for key in ("packed_codes", "radius_codes", "radius_grid", "codebook",
                                                     "permutation")], n).to(dtype)
    for bias in (None, torch.randn(n, generator=gen, device="cuda").to(dtype), torch.randn(n, generator=gen, device="cuda")):
        with torch.no_grad():
            got = SAGELinear(packed, n, bias)(x)
        want = plain if bias is None else plain + bias
        assert got.dtype == want.dtype and torch.equal(got, want)


@pytest.mark.parametrize("rows", [17, 77, 513])
@pytest.mark.parametrize("widths", [(256, 129, 1024), (4096, 1024, 1024), (640, 640)])
def test_rows_of_several_linears_in_one_launch(rows, widths):
    """q/k/v-like groups side by side in one GEMM launch (with and without CTA pairs and K splits, permuted and
    pregathered inputs) against each linear alone."""
    import ctypes

    from sage_b200 import SAGELinear, _lib

    lib, k = _lib.load(), 1280
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, k, generator=gen, device="cuda").half()
    mats = [{key: value.cuda() for key, value in synthetic_sage(k, n, seed=7 + i).items()} for i, n in enumerate(widths)]
    for gathered in (True, False):
        array, keep, outs = (_lib.Problem * len(widths))(), [], []
        for i, (m, n) in enumerate(zip(mats, widths)):
            xi = x[:, m["permutation"].long()].contiguous() if gathered else x
            keep.append(xi)
            outs.append(torch.zeros(rows, n, dtype=torch.float16, device="cuda"))
            array[i] = _lib.Problem(xi.data_ptr(), m["packed_codes"].data_ptr(), m["radius_codes"].data_ptr(),
                                    m["radius_grid"].data_ptr(), m["codebook"].data_ptr(),
                                    None if gathered else m["permutation"].data_ptr(), outs[i].data_ptr(), rows, n, k,
                                    m["codebook"].shape[1])
        nbytes = lib.sageb200_linear_rows_workspace_bytes(array, len(widths))
        scratch = torch.zeros(max(nbytes, 256), dtype=torch.uint8, device="cuda")
        for _ in range(2):
            assert lib.sageb200_linear_rows(array, len(widths), ctypes.c_void_p(scratch.data_ptr()), nbytes, None) == 0
        for m, n, out in zip(mats, widths, outs):
            want = SAGELinear(m, n)(x).float()
            assert ((out.float() - want).norm() / want.norm()) < 1e-3
        assert not scratch[:65536].any() or nbytes == 0


@pytest.mark.parametrize("tokens,first,spare", [(128, 0, 0), (129, 0, 100), (200, 37, 0), (300, 0, 1), (513, 250, 64), (1100, 0, 0)])
@pytest.mark.parametrize("q_heads,kv_heads", [(15, 3), (16, 2)])
def test_prompt_attention_tiles(tokens, first, spare, q_heads, kv_heads):
    """Partial tiles of rows and of positions, a cache that starts before the prompt, and rows of the cache
    beyond the prompt that hold no numbers; scores that grow along the prompt (the running maximum moves)."""
    import ctypes

    from sage_b200 import _lib

    lib, vp = _lib.load(), lambda t: ctypes.c_void_p(t.data_ptr())
    gen = torch.Generator(device="cuda").manual_seed(tokens + q_heads)
    sequences, max_seq = 5, first + tokens + spare
    q = torch.randn(sequences * tokens, q_heads, 128, generator=gen, device="cuda").half()
    k = torch.randn(sequences, kv_heads, max_seq, 128, generator=gen, device="cuda")
    k = (k * torch.linspace(0.5, 4.0, max_seq, device="cuda")[:, None]).half()
    v = torch.randn(sequences, kv_heads, max_seq, 128, generator=gen, device="cuda").half()
    k[:, :, first + tokens:], v[:, :, first + tokens:] = float("nan"), float("inf")
    positions = torch.full((sequences,), first, dtype=torch.int32, device="cuda")
    out = torch.zeros_like(q)
    assert lib.sageb200_glue_prefill_attention(vp(q), vp(k), vp(v), vp(positions), vp(out), sequences, tokens, q_heads,
                                               kv_heads, 128, max_seq, None) == 0
    torch.cuda.synchronize()
    end = first + tokens
    qf = q.float().view(sequences, tokens, q_heads, 128).transpose(1, 2)
    kf, vf = (t[:, :, :end].float().repeat_interleave(q_heads // kv_heads, dim=1) for t in (k, v))
    mask = torch.arange(end, device="cuda")[None, :] <= first + torch.arange(tokens, device="cuda")[:, None]
    scores = (qf @ kf.transpose(-1, -2) / 128 ** 0.5).masked_fill(~mask, float("-inf"))
    want = (scores.softmax(-1) @ vf).transpose(1, 2)
    got = out.float().view(sequences, tokens, q_heads, 128)
    assert torch.isfinite(got).all()
    assert ((got - want).norm() / want.norm()) < 1e-3
    assert (got - want).abs().max() < 1e-2


@pytest.mark.parametrize("tokens", [1, 3, 64, 85])
@pytest.mark.parametrize("q_heads,kv_heads", [(5, 1), (16, 4)])
def test_prompt_norm_and_rotation(tokens, q_heads, kv_heads):
    """Prompt rows, eight lanes per head (partial blocks, a cache that ends inside the prompt): bit for bit what a
    warp per head writes."""
    import ctypes

    from sage_b200 import _lib

    lib, vp = _lib.load(), lambda t: ctypes.c_void_p(t.data_ptr())
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device="cuda").half()
    sequences, first = 2, 5
    max_seq, rows = first + tokens - tokens // 8, sequences * tokens
    q, k, v = rand(rows, q_heads, 128), rand(rows, kv_heads, 128), rand(rows, kv_heads, 128)
    weights, tables = [rand(128), rand(128)], [rand(max_seq, 64), rand(max_seq, 64)]
    positions = torch.full((sequences,), first, dtype=torch.int32, device="cuda")
    results = []
    for shift in (0, 2):  # (an address that is not 16-byte aligned takes the warp-per-head kernel)
        qs = torch.zeros(q.numel() + 8, dtype=torch.float16, device="cuda")[shift:shift + q.numel()]
        qs.copy_(q.flatten())
        caches = [torch.zeros(sequences, kv_heads, max_seq, 128, dtype=torch.float16, device="cuda") for _ in range(2)]
        assert lib.sageb200_glue_prefill_qk_norm_rope_cache(
            vp(qs), vp(k), vp(v), vp(weights[0]), vp(weights[1]), vp(tables[0]), vp(tables[1]), vp(positions), vp(caches[0]),
            vp(caches[1]), sequences, tokens, q_heads, kv_heads, 128, max_seq, 1e-6, None) == 0
        results.append([qs.clone(), *caches])
    for one, two in zip(*results):
        assert torch.equal(one, two) and one.any()


@pytest.mark.parametrize("splits", [1, 2, 8])
@pytest.mark.parametrize("q_heads,kv_heads", [(4, 1), (5, 1), (2, 2)])
def test_decode_attention_tiles_and_rounds(splits, q_heads, kv_heads):
    """Contexts at the edges of the tiles of eight positions and of the rounds of a warp's ring, scores that grow along
    the context, and cache rows beyond it that hold no numbers, against an FP32 reference."""
    import ctypes

    from sage_b200 import _lib

    lib, vp = _lib.load(), lambda t: ctypes.c_void_p(t.data_ptr())
    gen = torch.Generator(device="cuda").manual_seed(splits + q_heads)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device="cuda").half()
    max_seq = 700
    positions = torch.tensor([0, 6, 7, 8, 63, 64, 65, 127, 128, 191, 255, 256, 511, 698, 699], dtype=torch.int32, device="cuda")
    rows = positions.numel()
    q, k, v = rand(rows, q_heads, 128), rand(rows, kv_heads, 128), rand(rows, kv_heads, 128)
    ones, cos, sin = torch.ones(128, device="cuda").half(), torch.ones(max_seq, 64, device="cuda").half(), torch.zeros(max_seq, 64, device="cuda").half()
    kc = (torch.randn(rows, kv_heads, max_seq, 128, generator=gen, device="cuda") *
          torch.linspace(0.2, 3.0, max_seq, device="cuda")[:, None]).half()
    vc = rand(rows, kv_heads, max_seq, 128)
    for r, p in enumerate(positions.tolist()):
        kc[r, :, p:], vc[r, :, p:] = float("nan"), float("inf")
    out = torch.zeros_like(q)
    assert lib.sageb200_glue_attention_step(vp(q), vp(k), vp(v), vp(ones), vp(ones), vp(cos), vp(sin), vp(positions), vp(kc),
                                            vp(vc), vp(out), rows, q_heads, kv_heads, 128, max_seq, splits, 1e-6, None) == 0
    torch.cuda.synchronize()
    norm = lambda x: (x.float() * torch.rsqrt(x.float().square().mean(-1, keepdim=True) + 1e-6)).half().float()
    for r, p in enumerate(positions.tolist()):
        keys, values = kc[r, :, :p + 1].float(), vc[r, :, :p + 1].float()
        keys, values = (x.repeat_interleave(q_heads // kv_heads, dim=0) for x in (keys, values))
        weights = (torch.einsum("hd,hpd->hp", norm(q[r]), keys) / 128 ** 0.5).softmax(-1)
        want = torch.einsum("hp,hpd->hd", weights, values)
        assert (out[r].float() - want).abs().max() < 4e-3, p


@pytest.mark.parametrize("rows,n,k", [(33, 19456, 1280), (65, 19000, 640), (520, 9729, 512), (1024, 19456, 512), (40, 25600, 2048)])
def test_gemm_with_a_split_rest(rows, n, k):
    """Grids of one full wave and a rest whose tiles alone are split along K (with and without pairs of CTAs, a partial
    row block and token block in the rest), repeatable, against a matmul on the dense weights."""
    from sage_b200 import SAGELinear

    packed = {key: value.cuda() for key, value in synthetic_sage(k, n, seed=rows).items()}
    x = torch.randn(rows, k, generator=torch.Generator(device="cuda").manual_seed(n), device="cuda").half()
    module = SAGELinear(packed, n)
    got = module(x)
    weight = sage_dequantize(packed["packed_codes"], packed["radius_codes"], packed["radius_grid"], packed["codebook"],
                             packed["permutation"], n).float()
    want = x.float() @ weight.T
    assert ((got.float() - want).norm() / want.norm()) < 1e-3
    assert (got.float() - want).abs().max() < 0.02 * want.abs().max()
    assert torch.equal(module(x), got)


@pytest.mark.parametrize("rows", [9, 16])
@pytest.mark.parametrize("fused", [False, True])
def test_gate_and_up_one_after_another(rows, fused):
    """Two problems whose shares of the device would cut K run on the whole device in turn, behind one staging
    launch: each as alone, bit for bit."""
    from sage_b200.ops import sage_grouped

    k, n = 2560, 9728
    mats = [{key: value.cuda() for key, value in synthetic_sage(k, n, seed=3 + i).items()} for i in range(2)]
    names = ("packed_codes", "radius_codes", "radius_grid", "codebook", "permutation")
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x, delta = (torch.randn(rows, k, generator=gen, device="cuda").half() for _ in range(2))
    weight = torch.randn(k, generator=gen, device="cuda").half()
    residuals = [torch.empty_like(x) for _ in range(3)]
    activation = lambda i: (1, 1e-6, x, delta, weight, residuals[i]) if fused else None
    problems = [(x, *[m[name] for name in names]) for m in mats]
    both = sage_grouped(problems, [n, n], activation(0))
    for i in range(2):
        (alone,) = sage_grouped(problems[i:i + 1], [n], activation(1 + i))
        assert torch.equal(both[i], alone)
    if fused:
        assert torch.equal(residuals[0], x + delta)


@pytest.mark.parametrize("rows,edge", [(1, 24), (2, 16), (8, 16), (16, 16)])
def test_expert_blocks_on_both_sides_of_the_rule(rows, edge):
    """Grouped launches below `edge` blocks, two launches from there: both within FP16 rounding of FP64 on the dense
    weights (weights, gate, up, activation and result are each rounded once: 5 * 2^-11 / sqrt(3) = 1.4e-3 at most)."""
    from sage_b200.experts import SAGEExperts, expert_slice, synthetic_expert_stack

    hidden, inter = 512, 384
    shapes = ((hidden, inter), (hidden, inter), (inter, hidden))
    stacks = [synthetic_expert_stack(k, n, edge, 51 + j, "cuda") for j, (k, n) in enumerate(shapes)]
    module = SAGEExperts(*stacks)
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(edge, rows, hidden, generator=gen, device="cuda").half()
    names = ("packed_codes", "radius_codes", "radius_grid", "codebook", "permutation")
    for blocks in (edge - 1, edge):
        got = module.forward_blocks(x[:blocks], torch.arange(blocks, dtype=torch.int32, device="cuda")).double()
        for b in (0, blocks - 1):
            gate, up, down = (sage_dequantize(*[expert_slice(stack, b)[key] for key in names], n).double()
                              for stack, (_, n) in zip(stacks, shapes))
            want = (torch.nn.functional.silu(x[b].double() @ gate.T) * (x[b].double() @ up.T)) @ down.T
            assert ((got[b] - want).norm() / want.norm()) < 1.4e-3


@pytest.mark.parametrize("experts,first,top_k", [(1, 0, 1), (3, 2, 2), (8, 0, 8), (40, 5, 5)])
@pytest.mark.parametrize("foreign", [False, True])
def test_experts_on_both_sides_of_the_slot_rule(experts, first, top_k, foreign):
    """One problem per slot up to 32 slots, sorted by expert beyond: tokens on both sides, one expert for all of them,
    experts of other ranks and empty slots (a share of zero), against FP64 on the dense weights."""
    from sage_b200.experts import SAGEExperts, expert_slice, synthetic_expert_stack

    hidden, inter = 256, 384
    shapes = ((hidden, inter), (hidden, inter), (inter, hidden))
    stacks = [synthetic_expert_stack(k, n, experts, 61 + j, "cuda", first=first) for j, (k, n) in enumerate(shapes)]
    module = SAGEExperts(*stacks, first_expert=first)
    names = ("packed_codes", "radius_codes", "radius_grid", "codebook", "permutation")
    dense = [[sage_dequantize(*[expert_slice(stack, e)[key] for key in names], n).double() for e in range(experts)]
             for stack, (_, n) in zip(stacks, shapes)]
    for tokens in sorted({2, 32 // top_k, 32 // top_k + 1, 60}):
        gen = torch.Generator(device="cuda").manual_seed(tokens)
        x = torch.randn(tokens, hidden, generator=gen, device="cuda").half()
        ids = torch.stack([torch.randperm(experts, generator=gen, device="cuda")[:top_k] for _ in range(tokens)]) + first
        ids = ids.to(torch.int32)
        if foreign:
            ids[0], ids[1, 0], ids[-1, -1] = first + experts, -1, first - 1
        weights = torch.rand(tokens, top_k, generator=gen, device="cuda")
        got = module(x, ids, weights, foreign_experts=foreign).double()
        want = torch.zeros_like(got)
        for t in range(tokens):
            for j in range(top_k):
                e = int(ids[t, j]) - first
                if 0 <= e < experts:
                    act = torch.nn.functional.silu(x[t].double() @ dense[0][e].T) * (x[t].double() @ dense[1][e].T)
                    want[t] += weights[t, j].double() * (act @ dense[2][e].T)
        # (rounded once each: weights, gate, up, activation, the slot's result, the mix: 6 * 2^-11 / sqrt(3) at most)
        assert (got - want).norm() <= 1.7e-3 * want.norm(), tokens
        if foreign:
            assert not got[0].any()
