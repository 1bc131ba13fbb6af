"""The step tables of bench.py --design: every attention kernel that a model's parts launch has its line."""
import glob
import os
import re

import bench

ROOT = os.path.dirname(os.path.abspath(bench.__file__))


def test_every_attention_of_the_parts_is_timed():
    used = set()
    for path in glob.glob(os.path.join(ROOT, "rllm_b200", "parts", "*.py")):
        with open(path) as f:
            used |= set(re.findall(r"ops\.(\w*attention\w*)\(", f.read()))
    used = {n for n in used if not n.endswith(("_takes", "_pays")) and not n.startswith("use_")}
    # the CUDA-core forms belong to the 32-bit path, which the tables do not run
    used -= {"attention_simt", "latent_attention_simt"}
    assert "latent_attention_tcgen05" in used and used <= set(bench.STEP_KERNELS), used - set(bench.STEP_KERNELS)
