"""The rules beside pdl_wait / pdl_release in xb_common.cuh, read off the kernels' source: a kernel that may begin before the one
before it has ended waits ahead of any exit, and releases the next one only after its own tensor memory has been allocated (the
next kernel may allocate while it waits, and the two would wait for one another)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "x-deeplearning_b200", "csrc")


def _sources():
    out = {}
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(f).read())
        out[os.path.basename(f)] = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return out


def _kernels():
    """name -> body of every __global__ function"""
    found = {}
    for text in _sources().values():
        for m in re.finditer(r"__global__", text):
            name = None
            i = m.end()
            # the kernel's name is the identifier before the parameter list that the body follows
            for n in re.finditer(r"([A-Za-z_]\w*)\s*\(", text[i:i + 600]):
                if n.group(1) not in ("__launch_bounds__", "__cluster_dims__"):
                    name, i = n.group(1), i + n.end() - 1
                    break
            depth = 0
            while True:                                       # end of the parameter list
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
                if depth == 0:
                    break
            while text[i] not in "{;":
                i += 1
            if text[i] == ";":
                continue
            start, depth = i, 0
            while True:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
                if depth == 0:
                    break
            found[name] = text[start:i]
    return found


def _launched_early():
    names = set()
    for text in _sources().values():
        for m in re.finditer(r"launch_dependent\(([^;]*?)[,<]", text):
            if not m.group(1).startswith("void"):
                names.update(re.findall(r"\b(\w+_kernel)\b", m.group(0)))
        for m in re.finditer(r"launch_dependent\(\w+ \? (\w+)<", text):
            names.add(m.group(1))
        if "cudaLaunchAttributeProgrammaticStreamSerialization" in text:
            names.update(re.findall(r"cudaLaunchKernelEx\(&cfg, (\w+_kernel)<", text))
    return names


def test_kernels_launched_early_wait_before_any_exit():
    kernels, early = _kernels(), _launched_early()
    assert {"pool_fast_kernel", "gemm_umma_kernel", "gemm_umma_pair_kernel", "din_att_tc_kernel", "augru_tc_kernel", "gru_kernel",
            "copy2d_convert_kernel", "din_tower_tc_kernel", "route_one_kernel"} <= early and len(early) >= 40, sorted(early)
    for name in early:
        body = kernels[name]
        wait = re.search(r"\bpdl_(begin|wait)\(\)", body)
        assert wait, "%s is launched early and never waits" % name
        assert not re.search(r"\breturn\b", body[: wait.start()]), "%s can end before it has waited" % name
        # at the top level of the body: no thread goes past it
        assert body[: wait.start()].count("{") - body[: wait.start()].count("}") == 1, name


def test_tensor_memory_is_allocated_before_the_next_kernel_is_released():
    checked = 0
    for name, body in _kernels().items():
        release = re.search(r"\bpdl_(begin|release)\(\)", body)
        alloc = re.search(r"\btmem_alloc(_pair)?\(", body)
        if release and alloc:
            assert alloc.start() < release.start(), "%s releases the next kernel before its tensor memory is allocated" % name
            # every thread of the block has met the one that allocates
            assert "__syncthreads()" in body[alloc.start(): release.start()], name
            checked += 1
    assert checked >= 4


def test_a_cluster_that_shares_an_attention_tile_has_its_sm_to_itself():
    text = _sources()["xb_din_attention_tc.cuh"]
    kb = int(re.search(r"TC_CLUSTER_SMEM = (\d+) \* 1024", text).group(1))
    assert 2 * kb > 228 and kb <= 220
    assert re.search(r"p\.split > 1 \? std::max<size_t>\(\(size_t\)L\.total, TC_CLUSTER_SMEM\)", text)
