"""Kernels that overlap the tail of the one in front (griddepcontrol.wait): what that kernel writes is not loaded through __restrict__ or __ldg.
Such loads count as invariant, so the compiler may move them ahead of the wait, and they would then read the rows of an earlier call.
A race that a run need not show, so the sources are what is checked: in every kernel that waits, the __restrict__ parameters are weights and
tables that were complete before the chain began, or buffers that the kernel only writes, and __ldg takes only the former."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vla_cpp_b200", "csrc")

INVARIANT = {  # kernel -> weights, biases, modulations, rotation tables
    "adarms_norm_kernel": {"mod"}, "adarms_norm_vec_kernel": {"mod"}, "action_in_kernel": {"w_ain", "b_ain"}, "state_token_kernel": {"w_sp", "b_sp"},
    "euler_kernel": set(), "splitk_reduce_kernel": {"colscale", "bias"}, "f32_skinny_linear_kernel": {"W", "bias"}, "f32_layernorm_kernel": {"w", "b"},
    "norm_quant_kernel": {"w"}, "norm_quant_vec_kernel": {"w"}, "rope_split_kernel": {"cos_t", "sin_t"}, "rope_split_vec_kernel": {"cos_t", "sin_t"},
    "rope_split_f32_kernel": {"cos_t", "sin_t"},
    "vit_ln_quant_kernel": {"add_bias", "ln_w", "ln_b"}, "vit_ln_quant_rows_kernel": {"add_bias", "ln_w", "ln_b"},
    "vit_split_heads_kernel": {"bq", "bk", "bv"}, "vit_merge_quant_kernel": set(), "vit_gelu_quant_kernel": {"bias"}, "vit_quant_rows_kernel": set(),
    "ternary_gemv_kernel": {"Wp", "ws"}, "ternary_gemm_tc_kernel": {"Wp", "ws"}, "ternary_gemm_pair_kernel": {"Wp", "ws"},
    "layernorm_vec_kernel": {"w", "b"},
}
WRITTEN = {"out", "acc_out", "a", "a_f32", "y", "h", "hb", "q_out", "s_out", "out_bf", "k_pages", "v_pages", "q", "kp", "vp"}  # and never read
WRITTEN_ONLY_HERE = {"h": {"state_token_kernel"}, "a": {"action_in_kernel"}, "q": {"vit_split_heads_kernel"}}  # names that are inputs elsewhere
LDG = {"w", "W", "Wp", "wbase", "wa", "wb", "wr", "ln_w", "ln_b", "add_bias", "mod", "cos_t", "sin_t", "cp", "sp", "cs_row", "sn_row", "colscale", "bias", "b"}


def strip_comments(text):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def body_at(text, brace):
    depth = 0
    for i in range(brace, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[brace:i + 1]
    raise AssertionError("unbalanced braces")


def functions(text, qualifier):
    for m in re.finditer(qualifier, text):
        end = re.compile(r"[{;]").search(text, m.end())
        if not end or text[end.start()] == ";":
            continue
        head = re.sub(r"__(?:launch_bounds|cluster_dims)__\s*\((?:[^()]|\([^()]*\))*\)", "", text[m.end():end.start()])
        name, params = re.search(r"(\w+)\s*\((.*)\)\s*$", head, flags=re.S).groups()
        yield name, params, body_at(text, end.start())


def calls(body, names):
    return any(re.search(r"\b%s\s*(?:<[^;(]*>)?\s*\(" % n, body) for n in names)


def waiting_kernels():
    found = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = strip_comments(open(path).read())
        bodies = {n: b for n, _, b in functions(text, r"__device__ __forceinline__") if "pdl_wait" in b}
        for name, params, body in functions(text, r"__global__"):
            if "pdl_wait" in body or calls(body, bodies):
                found[name] = (params, body + "".join(b for n, b in bodies.items() if calls(body, [n])))
    return found


KERNELS = waiting_kernels()


def test_the_parser_sees_the_kernels():
    assert len(KERNELS) >= 30 and set(INVARIANT) <= set(KERNELS), set(INVARIANT) - set(KERNELS)


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_only_weights_and_tables_are_read_as_invariant(name):
    params, body = KERNELS[name]
    for p in params.split(","):
        if "__restrict__" in p:
            arg = re.search(r"(\w+)\s*$", p).group(1)
            ok = arg in INVARIANT.get(name, set())
            if not ok and "const" not in p:
                ok = arg in WRITTEN and name in WRITTEN_ONLY_HERE.get(arg, {name})
            assert ok, f"{name}: {arg} may be the output of the kernel in front"
    for arg in re.findall(r"__ldg\(((?:[^()]|\((?:[^()]|\([^()]*\))*\))*)\)", body):
        roots = set(re.findall(r"(?<![\w.])(?:p\.)?([A-Za-z_]\w*)", arg))
        assert roots & LDG, f"{name}: __ldg({arg})"
