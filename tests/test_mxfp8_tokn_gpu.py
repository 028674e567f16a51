"""Token-N mxfp8 kernels (routed rows on the N side of the block-scaled MMA): expert sizes at the edges of a work item.

The reference is the same FFN in fp64 on the dequantised operands, with the activation re-quantised as the kernels do.
"""
import pytest
import torch

from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def run(counts, K, N, bpc=1, T_extra=0):
    """counts[e] routed rows for expert e, one expert per token; T_extra tokens are routed nowhere (expert id E)."""
    import prime_flash_moe_b200 as P
    from prime_flash_moe_b200 import capi
    E, T = len(counts), sum(counts) + T_extra
    g = torch.Generator().manual_seed(K + N + T)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16)
    # rows and blocks of different scale: a scale taken from another row, block or k-step shows
    spread = lambda r, c: torch.exp2(torch.randint(-3, 4, (r, c // 32), generator=g).float()).repeat_interleave(32, 1)
    x = (x * spread(T, K)).to(torch.bfloat16)
    w1 = ((torch.randn(E * N, K, generator=g) / K ** 0.5) * spread(E * N, K)).to(torch.bfloat16).view(E, N, K)
    w2 = ((torch.randn(E * K, N // 2, generator=g) / (N // 2) ** 0.5) * spread(E * K, N // 2)).to(torch.bfloat16).view(E, K, N // 2)
    q = [O.quantize_mx(t) for t in (x, w1, w2)]
    dx, dw1, dw2 = (O.dequantize_mx(*t).double() for t in q)
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)] +
                    [torch.full((T_extra,), E, dtype=torch.int32)])
    ids = ids[torch.randperm(T, generator=g)].view(T, 1).contiguous()
    wts = torch.rand(T, 1, generator=g) + 0.5
    s, e, n = capi.moe_align(ids.to(DEV), E, 128, bpc)
    out = torch.full((T, K), float("nan"), dtype=torch.bfloat16, device=DEV)
    capi.fused_moe_mxfp8(q[0][0].to(DEV), q[0][1].to(DEV), q[1][0].to(DEV), P.pack_scales_blocked(q[1][1]).to(DEV),
                         q[2][0].to(DEV), P.pack_scales_blocked(q[2][1]).to(DEV), s, e, n, wts.to(DEV), out, 1, bpc=bpc)
    torch.cuda.synchronize()
    assert capi.device_status() == 0
    ref = torch.zeros(T, K, dtype=torch.float64)
    for ex in range(E):
        rows = (ids[:, 0] == ex).nonzero().flatten()
        gu = dx[rows] @ dw1[ex].t()
        act = (torch.nn.functional.silu(gu[:, :N // 2]) * gu[:, N // 2:]).float()
        if len(rows):
            act = O.dequantize_mx(*O.quantize_mx(act))
        ref[rows] = wts[rows].double() * (act.double() @ dw2[ex].t())
    err = (out.double().cpu() - ref).norm(dim=1) / ref.norm(dim=1).clamp_min(1e-30)
    # bf16 result: 2^-9. An activation next to an e4m3 rounding boundary may go the other way, 2^-3 of its value: one of
    # N / 2 >= 128 of them, whose w2 column may be 2^3 times the others' rms / 2.8: 2^-3 * 2.8 / sqrt(128) < 2^-5 of the row
    live = err[ids[:, 0] < E]
    assert live.max() < 2 ** -5 and live.square().mean().sqrt() < 2 ** -8, (float(err.max()), int(err.argmax()))
    assert torch.equal(out.cpu()[ids[:, 0] == E], torch.zeros(T_extra, K, dtype=torch.bfloat16))


@pytest.fixture(autouse=True)
def token_n(monkeypatch):
    monkeypatch.setenv("PMOE_TOKN", "1")


# few rows per expert: pieces of at most 64 rows, else of at most 192
@pytest.mark.parametrize("bpc", [1, 2])
@pytest.mark.parametrize("counts", [(1, 0, 2, 0), (31, 32, 33), (63, 65, 0, 1), (95, 97, 60), (127, 128, 129),
                                    (191, 192, 193), (0, 385, 300), (577, 1, 0)])
def test_expert_sizes_at_item_edges(counts, bpc):
    run(counts, 512, 512, bpc, T_extra=3)


# one tile a CTA pair, an odd number of 128-wide tiles, more k-steps than ring slots, K % 512 == 256, several rounds of tiles
@pytest.mark.parametrize("K,N", [(512, 256), (768, 768), (2048, 256), (1280, 2816)])
@pytest.mark.parametrize("counts", [(5, 0, 20), (200, 130, 7), (800, 640, 1000)])
def test_matrix_sizes_at_tile_edges(counts, K, N):
    run(counts, K, N)
