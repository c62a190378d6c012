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


# `const __restrict__` parameters of kernels that wait for the one in front: a model's weights and tables, which no kernel of a pass writes
WEIGHTS = {
    "linear_rows_vec_kernel": "W bias", "linear_one_row_kernel": "W bias", "linear_rows_kernel": "W bias", "linear_tiled_kernel": "W bias",
    "linear_batched_rows_kernel": "W", "embed_tokens_kernel": "table", "layernorm_kernel": "gamma beta", "rmsnorm_kernel": "gamma",
    "rmsnorm_row_kernel": "gamma", "layernorm_rows_kernel": "gamma beta", "gated_group_rmsnorm_kernel": "gamma", "gated_group_rmsnorm_vec_kernel": "gamma",
    "embed_rows_kernel": "table", "rms_scalar_kernel": "g vec", "rms_scalar_reg_kernel": "g vec", "rms_weight_kernel": "w", "rms_weight_reg_kernel": "w",
    "embed_norm_kernel": "table w", "embed_norm_reg_kernel": "table w", "polynorm_kernel": "bias coef", "embed_bigram_kernel": "table bigram",
    "latent_append_kernel": "gamma", "causal_conv_kernel": "w bias", "token_shift_mix_kernel": "mu", "latent_rot_append_kernel": "gamma table",
    "vit_embed_ln_kernel": "cls pos gamma beta",
}
READ_ONLY = {"io.gamma", "tab", "ep.w_scale"}   # what __ldg reads: norm weights, cosines and sines, scales of weights


def waiting_parameters(src):
    """(kernel, its `const __restrict__` parameters, what it reads by __ldg) of every kernel that waits for the one in front of it"""
    src = re.sub(r"//[^\n]*|/\*.*?\*/", "", src, flags=re.S)
    for m in re.finditer(r"__global__\b", src):
        at = src.index("{", m.end())
        head, body = src[m.end():at], next(body for _, body in kernels(src[m.start():]))
        if re.search(r"\bpdl_(wait|enter)", body):
            yield (re.findall(r"(\w+_kernel)\b", head)[0], set(re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", head)),
                   set(re.findall(r"__ldg\((?:reinterpret_cast<[^>]*>\()?([\w.]+)", body)))


def test_rows_that_other_kernels_write_are_not_read_as_constants(repo_root):
    """The compiler may move a load through a `const __restrict__` parameter in front of griddepcontrol.wait, and then reads what the kernel in front
    has not written yet."""
    seen = 0
    for path in glob.glob(os.path.join(repo_root, "llava-plus-codebase_b200", "csrc", "*.cu")):
        for name, params, ldg in waiting_parameters(open(path).read()):
            seen += 1
            assert params <= set(WEIGHTS.get(name, "").split()), f"{os.path.basename(path)}: {name} reads {params} as constants"
            assert ldg <= READ_ONLY, f"{os.path.basename(path)}: {name} reads {ldg} as constants"
    assert seen >= 60


# conditions around a __syncthreads of one line, the same in every thread of a block: sizes and modes of the launch
UNIFORM = {"S > 1", "MODE == SCAN_SSD || MODE == SCAN_HGRN2 || p.prepared == 0"}


def test_block_barriers_are_reached_by_the_whole_block_at_one_place(repo_root):
    """__syncthreads asks for all threads of the block at the same call. Warps that meet at different places use a barrier by number (bar.sync)."""
    seen = 0
    for path in glob.glob(os.path.join(repo_root, "llava-plus-codebase_b200", "csrc", "*.cu")):
        src = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        for m in re.finditer(r"__syncthreads\(\)", src):
            seen += 1
            line = src[:m.start()].rsplit("\n", 2)
            cond = re.search(r"\bif (?:constexpr )?\((.*)\)\s*(?:\{[^}]*)?$", line[-1])
            if cond is None and re.search(r"\belse\s*(?:\{[^}]*)?$", line[-1]):
                cond = re.search(r"\bif \((.*?)\) [^;]*;\s*$", line[-2])
            assert cond is None or cond.group(1) in UNIFORM, f"{os.path.basename(path)}: a barrier behind if ({cond.group(1)})"
    assert seen >= 50


def test_pairs_meet_before_they_take_and_before_they_release_tensor_memory(repo_root):
    """Tensor memory of a CTA pair (cta_group::2) is taken and released by both CTAs. A CTA may start long before its peer, so the pair meets in front of the
    allocation; it meets in front of the release as its products are done by one of them."""
    seen = 0
    for path in glob.glob(os.path.join(repo_root, "llava-plus-codebase_b200", "csrc", "*.cu")):
        for name, body in kernels(open(path).read()):
            take, free = re.search(r"\btmem_alloc_2sm\(", body), re.search(r"\btmem_dealloc_2sm\(", body)
            if take is None:
                continue
            seen += 1
            meet = r"\bcluster_sync\(\)"
            assert re.search(meet, body[:take.start()]), f"{os.path.basename(path)}: {name} takes tensor memory before its pair has met"
            assert len(re.findall(meet, body[take.end():free.start()])) >= 2, f"{os.path.basename(path)}: {name} releases tensor memory before its pair has met"
    assert seen >= 1
