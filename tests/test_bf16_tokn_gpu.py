"""Token-N bf16 kernels (routed rows on the N side of the MMA): expert sizes at the edges of a work item.

The reference is the same FFN in fp64; the kernels round the activation and the result to bf16 (2^-9 relative each).
"""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def reference(x, w1, w2, ids, wts):
    """Expert FFN of every token (one expert per token, ids >= E: none) in fp64."""
    E, N = w1.shape[:2]
    ref = torch.zeros(x.shape, dtype=torch.float64)
    for e in range(E):
        rows = (ids[:, 0] == e).nonzero().flatten()
        gu = x[rows].double() @ w1[e].double().t()
        act = torch.nn.functional.silu(gu[:, :N // 2]) * gu[:, N // 2:]
        ref[rows] = wts[rows].double() * (act @ w2[e].double().t())
    return ref


def check(out, ref):
    """Row by row: one norm over all rows does not see a few lost ones."""
    err = (out.double().cpu() - ref).norm(dim=1) / ref.norm(dim=1).clamp_min(1e-30)
    assert err.max() < 2 ** -7, (float(err.max()), int(err.argmax()))     # two bf16 roundings (activation, result)


def run(counts, K, N, bpc, T_extra=0):
    """counts[e] routed rows for expert e, one expert per token; T_extra tokens are routed nowhere (expert id E)."""
    from prime_flash_moe_b200 import capi
    E, T = len(counts), sum(counts) + T_extra
    g = torch.Generator().manual_seed(K + N + T)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16)
    w1 = (torch.randn(E, N, K, generator=g) / K ** 0.5).to(torch.bfloat16)
    w2 = (torch.randn(E, K, N // 2, generator=g) / (N // 2) ** 0.5).to(torch.bfloat16)
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)] +
                    [torch.full((T_extra,), E, dtype=torch.int32)])
    ids = ids[torch.randperm(T, generator=g)].view(T, 1).contiguous()
    wts = torch.rand(T, 1, generator=g) + 0.5
    s, e, n = capi.moe_align(ids.to(DEV), E, 128, bpc)
    out = torch.full((T, K), float("nan"), dtype=torch.bfloat16, device=DEV)
    capi.fused_moe_bf16(x.to(DEV), w1.to(DEV), w2.to(DEV), s, e, n, wts.to(DEV), out, 1, bpc=bpc)
    torch.cuda.synchronize()
    assert capi.device_status() == 0
    check(out, reference(x, w1, w2, ids, wts))
    assert torch.equal(out.cpu()[ids[:, 0] == E], torch.zeros(T_extra, K, dtype=torch.bfloat16))


@pytest.fixture(autouse=True)
def token_n(monkeypatch):
    monkeypatch.setenv("PMOE_TOKN", "1")


# few rows per expert: pieces of at most 64 rows; many: of at most 256
@pytest.mark.parametrize("bpc", [1, 2])
@pytest.mark.parametrize("counts", [(1, 0, 2, 0), (31, 32, 33), (63, 65, 0, 1), (127, 128, 129), (255, 256, 257),
                                    (0, 513, 300), (640, 1, 0)])
def test_expert_sizes_at_item_edges(counts, bpc):
    run(counts, 256, 512, bpc, T_extra=3)


# runs of more row blocks than the planner looks at in one go (512); in the last two a run starts before such a chunk,
# covers all of it and ends where the next one begins, with a partly filled block
@pytest.mark.parametrize("counts", [(67000,), (66000, 3), (100, 65700, 40), (65536, 65536 + 1), (131044, 2000, 2000),
                                    (100, 130893, 300)])
def test_long_runs(counts):
    run(counts, 128, 256, 1)


@pytest.mark.parametrize("K,N", [(128, 256), (384, 256), (640, 768), (1152, 512)])   # one k-step pair, K % 256 == 128
def test_matrix_sizes_at_tile_edges(K, N):
    run((40, 0, 130, 7), K, N, 1)


# down kernel with bulk reductions (N >= 2048, 1024 rows per expert on average): pieces of 32 to 256 rows, K % 256 == 128,
# more k-steps than ring slots, chunks of one and of both epilogue groups
@pytest.mark.parametrize("counts,K,N", [((1024,), 128, 2048), ((3000, 0, 72), 384, 2304), ((1, 4095, 33, 0), 256, 2048),
                                        ((1900, 161, 1300, 735), 1152, 2048)])
def test_down_kernel_with_bulk_reductions(counts, K, N):
    from prime_flash_moe_b200 import capi
    assert capi.lib().pmoe_debug_tokn_bulk_down(sum(counts), N, len(counts), 1) == 1
    run(counts, K, N, 1)


def test_an_expert_seen_in_separate_runs_and_holes_inside_a_block():
    """A hand-made routing table: expert 0 in two separate runs, and a block whose rows are not contiguous."""
    from prime_flash_moe_b200 import capi
    K, N, E, T = 256, 512, 2, 300
    g = torch.Generator().manual_seed(1)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16)
    w1 = (torch.randn(E, N, K, generator=g) / 16).to(torch.bfloat16)
    w2 = (torch.randn(E, K, N // 2, generator=g) / 16).to(torch.bfloat16)
    table = torch.full((4, 128), -1, dtype=torch.int32)
    table[0] = torch.arange(128)
    table[1, :20] = torch.arange(128, 148)
    table[2, 5:128:2] = torch.arange(148, 210)         # holes
    table[3, :90] = torch.arange(210, 300)
    experts = torch.tensor([0, 1, 0, 0], dtype=torch.int32)
    wts = torch.rand(T, 1, generator=g) + 0.5
    out = torch.empty(T, K, dtype=torch.bfloat16, device=DEV)
    capi.fused_moe_bf16(x.to(DEV), w1.to(DEV), w2.to(DEV), table.view(-1).to(DEV), experts.to(DEV),
                        torch.tensor([512], dtype=torch.int32, device=DEV), wts.to(DEV), out, 1)
    torch.cuda.synchronize()
    assert capi.device_status() == 0
    ids = torch.zeros(T, 1, dtype=torch.int32)
    ids[128:148] = 1
    check(out, reference(x, w1, w2, ids, wts))


@pytest.mark.parametrize("listed_twice", [False, True])
@pytest.mark.parametrize("top_k,K", [(2, 2176), (3, 4096)])
def test_rows_gathered_token_by_token(top_k, K, listed_twice):
    """More than 64 MB of activations, gathered row by row inside the gate/up kernel; some pairs are routed nowhere, some
    tokens not at all; a hand-made table may list a pair in two rows. The row-M kernels give the expected result."""
    import os
    from prime_flash_moe_b200 import capi
    N, E = 256, 40
    T = (64 << 20) // (2 * K) + 5
    g = torch.Generator(device=DEV).manual_seed(K)
    x = torch.randn(T, K, generator=g, device=DEV, dtype=torch.bfloat16)
    w1 = torch.randn(E, N, K, generator=g, device=DEV, dtype=torch.bfloat16) * K ** -0.5
    w2 = torch.randn(E, K, N // 2, generator=g, device=DEV, dtype=torch.bfloat16) * (N // 2) ** -0.5
    ids = torch.rand(T, E + 3, generator=g, device=DEV).topk(top_k).indices.to(torch.int32)   # ids >= E: no expert
    ids[7] = E
    wts = torch.rand(T, top_k, generator=g, device=DEV)
    s, e, n = capi.moe_align(ids.contiguous(), E, 128, 1)
    if listed_twice:       # the first padding row of every block takes the pair of the block's first row
        table = s.view(-1, 128)
        fill = (table >= 0).sum(1)
        blocks = ((fill > 0) & (fill < 128)).nonzero().flatten()
        assert len(blocks) > E // 2
        table[blocks, fill[blocks]] = table[blocks, 0]
    ws = torch.empty(capi.lib().pmoe_fused_moe_bf16_workspace_bytes(T, K, N, s.numel(), 1) + 1024, dtype=torch.uint8,
                     device=DEV)
    ws = ws[-ws.data_ptr() % 1024:]
    outs = []
    for mode in ("1", "0"):
        os.environ["PMOE_TOKN"] = mode      # the fixture restores the variable
        ws.fill_(255)                       # NaN where nothing is written
        outs.append(capi.fused_moe_bf16(x, w1, w2, s, e, n, wts, torch.empty_like(x), top_k, workspace=ws).float())
    torch.cuda.synchronize()
    assert capi.device_status() == 0
    # row by row; each path rounds to bf16 at the activation, the products and at most top_k + 1 sums: independent errors
    # of 2^-9, sqrt(6) * 2^-9 < 2^-7 for each path
    err = (outs[0] - outs[1]).norm(dim=1) / outs[1].norm(dim=1).clamp_min(1e-30)
    assert err.max() < 2 ** -6, (float(err.max()), int(err.argmax()))
    assert not outs[0][7].any()


@pytest.mark.parametrize("counts", [(31, 0, 33), (257, 128, 5), (640, 70)])
def test_kept_pre_activations(counts):
    """gate | up of the routed rows in bf16, at the place of the row in the routing table."""
    from prime_flash_moe_b200 import capi
    K, N, E, T = 256, 768, len(counts), sum(counts)
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16)
    w1 = (torch.randn(E, N, K, generator=g) / 16).to(torch.bfloat16)
    w2 = (torch.randn(E, K, N // 2, generator=g) / 20).to(torch.bfloat16)
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)]).view(T, 1)
    wts = torch.rand(T, 1, generator=g) + 0.5
    s, e, n = capi.moe_align(ids.to(DEV), E, 128, 1)
    out, gate_up = capi.fused_moe_bf16_keep(x.to(DEV), w1.to(DEV), w2.to(DEV), s, e, n, wts.to(DEV),
                                            torch.empty(T, K, dtype=torch.bfloat16, device=DEV), 1)
    torch.cuda.synchronize()
    assert capi.device_status() == 0
    check(out, reference(x, w1, w2, ids, wts))
    rows = s.cpu().long()
    kept = gate_up.cpu()[rows >= 0].double()
    tok = rows[rows >= 0]
    ref = torch.stack([w1[ids[t, 0]].double() @ x[t].double() for t in tok])
    assert (kept - ref).norm() / ref.norm() < 2 ** -8      # one bf16 rounding
