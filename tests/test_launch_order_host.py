"""Order of set-up in the kernels that hold tensor memory, read from their source (no GPU: a kernel that gets it wrong may hang one)."""
import glob
import os
import re


def kernels(src):
    """(name, body) of every __global__ function of a file, comments taken out"""
    src = re.sub(r"//[^\n]*|/\*.*?\*/", "", src, flags=re.S)
    for m in re.finditer(r"__global__\b", src):
        at = src.index("{", m.end())
        depth, end = 1, at + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(src[end], 0)
            end += 1
        head = src[m.end():at]
        yield re.findall(r"(\w+_kernel)\b", head)[0], src[at:end]


def test_dependents_start_behind_the_allocation_of_tensor_memory(repo_root):
    """A dependent launch that allocates tensor memory waits for this kernel while it holds it. If it can be resident before this kernel has
    allocated, both wait for good: so the allocation and a barrier come first, then the trigger."""
    seen = 0
    for path in glob.glob(os.path.join(repo_root, "llava-plus-codebase_b200", "csrc", "*.cu")):
        for name, body in kernels(open(path).read()):
            alloc = re.search(r"\btmem_alloc\w*\(", body)
            if alloc is None:
                continue
            seen += 1
            starts = [m.start() for m in re.finditer(r"\bpdl_(trigger\w*|enter)\(", body)]
            if starts:   # (no trigger: dependents start when the kernel has ended)
                between = body[alloc.end():min(starts)] if min(starts) > alloc.start() else ""
                assert re.search(r"__syncthreads\(\)|cluster_sync\w*\(", between), f"{os.path.basename(path)}: {name} lets dependents start before its allocation"
    assert seen >= 8


def test_cluster_barriers_take_whole_warps(repo_root):
    """barrier.cluster in its aligned form needs every lane of a warp at the same instruction; behind a loop whose lanes leave at different turns only
    __syncwarp brings them there. So there is one function with the barrier, and it begins with that."""
    seen = 0
    for path in glob.glob(os.path.join(repo_root, "llava-plus-codebase_b200", "csrc", "*.cu*")):
        src = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        for m in re.finditer(r"barrier\.cluster\.arrive[\w.]*aligned", src):
            seen += 1
            assert re.search(r"__syncwarp\(\);\s*asm volatile\(\"$", src[:m.start()]), os.path.basename(path)
    assert seen >= 1
