"""Source-level rule for the dependent launches: a kernel that is launched with programmatic stream serialisation
(`launch_dependent`, `launch_dependent_if`) may start while the kernel before it still runs, so its body must contain
the wait that holds it back before the first access to global memory (`grid_dependency_wait`).  No GPU needed."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda_ltc_b200", "csrc")


def _sources():
    out = {}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh", ".h")):
            with open(os.path.join(CSRC, name)) as f:
                out[name] = f.read()
    return out


def _kernel_bodies(text):
    """name -> body for every __global__ function of a source file (brace matching)."""
    bodies = {}
    for m in re.finditer(r"__global__\s+void(?:\s+__launch_bounds__\([^)]*\))?\s+(\w+)\s*\(", text):
        i = text.index("{", m.end())
        depth, j = 1, i + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        bodies[m.group(1)] = text[i:j]
    return bodies


def _launched(text, bodies):
    """(launch, kernels) for every dependent launch of a source file.  A kernel picked at run time goes by a local name:
    it stands for every kernel named between its declaration and the launch."""
    spots = [(m, m.group(1)) for m in re.finditer(r"launch_dependent\(\s*([\w<>:, ]+?),\s*\S*(?:dim3|grid|rg)\b", text)]
    spots += [(m, m.group(1)) for m in re.finditer(r"launch_dependent_if\([^;]*?\),\s*([\w<>:, ]+?),\s*\S*(?:dim3|grid|gq|gk)\b", text)]
    spots += [(m, m.group(1)) for m in re.finditer(r"cudaLaunchKernelEx\(&cfg,\s*(\w+)", text)
              if "cudaLaunchAttributeProgrammaticStreamSerialization" in text]
    for m, name in spots:
        base = re.sub(r"<.*", "", name).strip()
        if base in bodies:
            yield m.group(0), {base}
            continue
        declared = text.rfind(f"auto {base} =", 0, m.start())
        assert declared >= 0, f"{m.group(0)}: {base} is neither a kernel nor a local name for one"
        named = set(re.findall(r"\b\w+_kernel\b", text[declared:m.start()])) & set(bodies)
        assert named, f"{m.group(0)}: no kernel found behind {base}"
        yield m.group(0), named


def test_every_dependent_launch_targets_a_kernel_that_waits():
    src = _sources()
    bodies = {}
    for text in src.values():
        bodies.update(_kernel_bodies(text))
    seen = set()
    for name, text in src.items():
        if name == "host_common.h":
            continue                                        # the helpers' own definitions
        found = list(_launched(text, bodies))
        # the pattern has to see every launch of the file
        direct = text.count("cudaLaunchKernelEx(") if "cudaLaunchAttributeProgrammaticStreamSerialization" in text else 0
        assert len(found) == len(re.findall(r"launch_dependent(?:_if)?\(", text)) + direct, name
        for launch, kernels in found:
            for k in kernels:
                assert "grid_dependency_wait()" in bodies[k], f"{name}: {k} is launched as a dependent kernel but never waits"
            seen |= kernels
    # kernels that are picked at run time or launched directly
    assert {"attn_fwd_tile_sm100_kernel", "gemm_bf16_sm100_kernel", "attn_decode_kernel", "pack_bf16_kernel",
            "gemm_splitk_reduce_kernel", "wide_softmax_fwd_rows_kernel", "attn_bwd_dkv_sm100_kernel"} <= seen


def test_waiting_kernels_touch_no_kernel_argument_memory_before_the_wait():
    """Before its wait a kernel may set up shared memory, barriers and tensor memory only: no pointer of the argument
    block is dereferenced there (the key lengths get a wait of their own where they are read early)."""
    for text in _sources().values():
        for name, body in _kernel_bodies(text).items():
            k = body.find("grid_dependency_wait()")
            if k < 0:
                continue
            before = body[:k]
            assert not re.search(r"\ba\.\w+\[|\bg\.\w+\[[^\]]*\]\s*[^;=]*;|__ldg\(|atomic\w+\(", before), name


def test_columns_that_two_warps_share_are_handed_over_with_fences():
    """The wider forward tile: P overwrites score columns that the row's other warp has loaded, so the meeting of the two
    lies between the two halves of a tensor-memory hand-over."""
    body = _kernel_bodies(_sources()["attn_fwd_sm100.cu"])["attn_fwd_tile_sm100_kernel"]
    steps = body[body.index("*xslot(j & 1, half) = mt;"):]
    order = [steps.index(s) for s in ("tc_fence_before_sync()", "meet()", "tc_fence_after_sync()", "tmem_st16(tP")]
    assert order == sorted(order)


def test_first_product_of_a_step_waits_for_every_warp_that_rescales():
    """The forward tile's products add to all columns of O: the barrier in front of a step's first product counts every math
    warp, and where a row's columns belong to two warps the second one arrives on it behind its rescale."""
    body = _kernel_bodies(_sources()["attn_fwd_sm100.cu"])["attn_fwd_tile_sm100_kernel"]
    assert "mbar_init(bar_p_full, L::kMathWarps)" in body
    steps = body[body.index("tmem_st16(tO + c0, o);"):]
    order = [steps.index(s) for s in ("if (half == 1) {", "tmem_wait_st();", "tc_fence_before_sync();", "mbar_arrive(bar_p_full);",
                                      "tmem_st16(tP")]
    assert order == sorted(order)
