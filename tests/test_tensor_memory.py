"""Kernels that wait for the kernel ahead of them while they hold tensor memory, beside kernels that still need theirs."""
import pytest
import torch

SM_SHARED, RESERVED = 228 * 1024, 1024  # bytes of an SM, and what the system takes of them for each CTA


def test_a_cta_with_all_of_the_tensor_memory_shares_no_sm_with_prompt_attention():
    """Counted on the host for every tile that a product of many tokens may have: with 512 columns taken, a CTA of prompt attention
    on the same SM would wait for the end of a product that waits for the end of the attention."""
    import kirai_b200  # noqa: F401
    from kirai_b200.csrc import ops

    lib = ops.library()
    for head_dim in (64, 128, 256):
        attention = lib.kirai_attention_prefill_tc_shared(head_dim)
        for row_tiles in (1, 2):
            for width in range(48 if row_tiles == 1 else 96, 257, 16):
                product = lib.kirai_gemm_bf16_many_shared(row_tiles, width)
                assert product <= 227 * 1024
                assert product + attention + 2 * RESERVED > SM_SHARED, (head_dim, row_tiles, width)


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,q_heads,width", [(1153, 64, 2880), (1665, 32, 2048), (769, 64, 4096)])
def test_a_product_of_many_tokens_behind_prompt_attention_over_narrow_heads(tokens, q_heads, width):
    """Heads of 64 columns, whose CTAs are the smallest that take tensor memory, and the products whose tiles of 128 x 208 have the
    smallest ring."""
    import kirai_b200  # noqa: F401
    from kirai_b200.csrc import ops

    assert ops.library().kirai_gemm_bf16_many_tile(tokens, width, 64 * q_heads, 0) == 1208  # (on 148 SMs)
    device, kv_heads, page = "cuda:0", 8, 16
    generator = torch.Generator().manual_seed(tokens)
    pages = -(-tokens // page)
    cache = torch.randn(pages, 2, kv_heads, page, 64, generator=generator).bfloat16().to(device)
    q = torch.randn(tokens, q_heads, 64, generator=generator).bfloat16().to(device)
    weight = (0.02 * torch.randn(width, 64 * q_heads, generator=generator)).bfloat16().to(device)
    table = torch.arange(pages, dtype=torch.int32, device=device).view(1, -1)
    start = torch.tensor([0, tokens], dtype=torch.int32, device=device)
    length = torch.tensor([tokens], dtype=torch.int32, device=device)
    tiled = ops.tile_weight(weight)
    results = []
    for _ in range(4):
        mixed = ops.attention_prefill(q, cache, table, start, length, tokens, None, 0.125)
        results.append((mixed, ops.linear_tcgen05(mixed, tiled, torch.float32)))
    ops.check_device_errors(torch.device(device))
    mixed, out = results[0]
    k = 64 * q_heads
    expected, size = mixed.double() @ weight.double().T, mixed.double().abs() @ weight.double().abs().T
    assert bool(((out.double() - expected).abs() <= 2 * k * 2.0 ** -24 * size).all())  # 32-bit sums of k products in any order
    for again in results[1:]:
        assert torch.equal(again[0], mixed) and torch.equal(again[1], out)
