"""Kernels start before the one ahead has ended (programmatic dependent launch): what that asks of their sources, read here as
text."""
import glob
import os
import re

import pytest

from rllm_b200.kernels import build

# arguments that no kernel of a step writes: the step's inputs, weights and constants
INPUTS = {"block_table", "q_start", "seq_lens", "slots", "inv_freq", "decay", "sink", "bias"}
WEIGHTS = {"embedding_kernel": {"table"}, "rmsnorm_kernel": {"w"}, "layernorm_kernel": {"w", "b", "c"}, "add_rows_kernel": {"c"},
           "add_row_bias_kernel": {"c"}, "gemm_small_m_kernel": {"W"}}
# read by asm statements alone (bulk copies, ld_cached16), which stay behind the wait
BY_ADDRESS = {"lightning_outputs_kernel": {"work"}, "gemm_small_m_kernel": {"x"}}


def kernels():
    """(file, name, parameters, body) of every kernel."""
    found = []
    for path in sorted(glob.glob(os.path.join(build.CSRC, "*.cu*"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"__global__\s+void\b", text):
            i = m.end()
            while True:                                    # attributes with arguments, then the name and its parameters
                head = re.compile(r"\s*(?:__cluster_dims__|__launch_bounds__)\s*\(").match(text, i)
                at = text.index("(", i)
                end, depth = at, 0
                while True:
                    depth += {"(": 1, ")": -1}.get(text[end], 0)
                    end += 1
                    if depth == 0:
                        break
                if not head:
                    break
                i = end
            name, params = text[i:at].strip(), text[at + 1:end - 1]
            start = text.index("{", end)
            if ";" in text[end:start]:
                continue                                   # a declaration
            stop, depth = start, 0
            while True:
                depth += {"{": 1, "}": -1}.get(text[stop], 0)
                stop += 1
                if depth == 0:
                    break
            found.append((os.path.basename(path), name, params, text[start:stop]))
    return found


def test_the_kernels_are_found():
    names = {k[1] for k in kernels()}
    assert len(names) > 60 and {"gemm_tcgen05_kernel", "gemm_tcgen05_pair_kernel", "lightning_act_kernel", "attention_decode_kernel"} <= names


@pytest.mark.parametrize("file,name,params,body", [k for k in kernels() if "pdl_wait" in k[3]], ids=lambda v: v if len(v) < 60 else "")
def test_what_the_kernel_ahead_wrote_is_not_declared_unwritten(file, name, params, body):
    """A ``const __restrict__`` parameter's loads may move ahead of the wait for the kernel ahead (common.cuh, pdl_fresh): such
    a parameter is an input of the step, or its pointer is made anew behind the wait."""
    fresh = set(re.findall(r"pdl_fresh\(\s*(?:\([^()]*\)\s*)?(\w+)", body))
    for args in re.findall(r"pdl_wait_on\(([^)]*)\)", body):
        fresh |= set(re.findall(r"\w+", args))
    for p in re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params):
        assert p in INPUTS | fresh | WEIGHTS.get(name, set()) | BY_ADDRESS.get(name, set()), f"{file}: {name}: {p}"


@pytest.mark.parametrize("file,name,params,body", [k for k in kernels() if "tcgen05.alloc" in k[3] and "pdl_launch" in k[3]],
                         ids=lambda v: v if len(v) < 60 else "")
def test_the_next_kernel_comes_in_behind_the_allocation_of_tensor_memory(file, name, params, body):
    """Else its CTAs may hold columns and wait for this kernel's end while a CTA of this kernel waits for columns."""
    assert body.index("tcgen05.alloc") < body.index("__syncthreads", body.index("tcgen05.alloc")) < body.index("pdl_launch"), f"{file}: {name}"
    assert body.index("pdl_wait") < body.index("pdl_launch")
