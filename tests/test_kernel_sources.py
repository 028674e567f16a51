"""Rules of the CUDA sources that no run can show."""
import re
from pathlib import Path

import prime_flash_moe_b200

CSRC = Path(prime_flash_moe_b200.__file__).parent / "csrc"

# Launched once init_kernel has passed its own wait, so whatever ran before the backward pass is complete, and that is all they
# take as constant.
COMPLETE_BEFORE = {"row_maps_kernel", "gather_token_rows_kernel"}
# files whose kernels are launched plainly
PLAIN = {"moe_ep.cu"}


def functions(text):
    """(name, parameters, body) of every __global__ or __device__ function defined in `text`."""
    text = re.sub(r"//[^\n]*|__launch_bounds__\([^()]*\)", "", text)
    for m in re.finditer(r"__(?:global|device)__[^;{}()]*?(\w+)\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params, rest = text[m.end():i - 1], text[i:].lstrip()
        if not rest.startswith("{"):
            continue
        start = j = text.index("{", i)
        depth = 0
        while True:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
            if depth == 0:
                break
        yield m.group(1), "__global__" in m.group(0), params, text[start:j]


def test_programmatic_dependents_read_no_constant_path():
    """Kernels launched as programmatic dependents may be resident while the kernel before them still writes. What that one
    writes they must not read through the non-coherent path, whose data has to be constant while the kernel runs: no `const T
    *__restrict__` parameter (the compiler may then choose that path by itself) and no `__ldg` in a kernel that waits for its
    primary, nor in the device functions it may call."""
    waiting, bad = set(), []
    for path in sorted(CSRC.glob("*.cu*")):
        for name, is_kernel, params, body in functions(path.read_text()):
            waits = "pdl_wait_primary()" in body or "griddepcontrol.wait" in body
            if is_kernel and waits:
                waiting.add(name)
            if path.name in PLAIN or name in COMPLETE_BEFORE or (is_kernel and not waits):
                continue
            if re.search(r"\bconst\b[^,]*\*\s*(const\s*)?__restrict__", params):
                bad.append(f"{path.name}: {name} takes a const __restrict__ pointer")
            if "__ldg(" in body:
                bad.append(f"{path.name}: {name} loads by __ldg")
    # the parser sees them: one of every file that launches programmatic dependents, and the exceptions
    assert {"plan_kernel", "moe_tokn_kernel", "live_items_kernel", "pair_items_kernel", "combine_dx_kernel", "route_topk_kernel",
            "quantize_mx_kernel", "moe_align_small_kernel", "moe_align_scatter_kernel", "gather_rows_mxfp8_kernel",
            "finalize_acc32_kernel"} | COMPLETE_BEFORE <= waiting
    assert not bad, "\n".join(bad)


def test_scopes_of_arrivals_in_the_peer_cta():
    """An arrival in the peer CTA releases at cluster scope where the wait acquires at cluster scope. The CTA-scope one hands
    over drained accumulators (after tcgen05.fence::before_thread_sync) and shared memory fenced to the async proxy only."""
    cluster, plain = set(), 0
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        assert ("mbar_wait_cluster(" in text) == ("mbar_arrive_cluster(" in text), path.name
        if "mbar_arrive_cluster(" in text:
            cluster.add(path.name)
        for m in re.finditer(r"mbar_arrive_peer_tcgen05\(", text):
            before = text[max(0, m.start() - 120):m.start()]
            assert "tc_fence_before();" in before or "fence_proxy_async_smem();" in before, (path.name, before)
            plain += 1
    assert cluster == {"moe_bf16.cu", "moe_mxfp8.cu"} and plain >= 4


def test_producers_wait_for_their_copies_in_flight():
    """A kernel whose TMA producer gives up a wait lets the copies already issued land before it ends."""
    seen = set()
    for path in sorted(CSRC.glob("*.cu")):
        for name, is_kernel, _, body in functions(path.read_text()):
            if is_kernel and "ST_TIMEOUT_EMPTY" in body and "tma_load" in body:
                seen.add(name)
                assert re.search(r"drain_(pair_)?fills\(|20000000ull", body), f"{path.name}: {name}"
    assert {"moe_tokn_kernel", "moe_up_dual_bf16_kernel", "moe_pair_bf16_kernel", "moe_pair_mxfp8_kernel", "moe_bwd_gemm_kernel",
            "moe_bwd_pair_kernel", "moe_fused_bf16_kernel"} <= seen
