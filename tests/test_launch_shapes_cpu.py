"""The launch shapes of the resource model are those of the kernels' sources."""
import re
from pathlib import Path

import pytest

from dew_b200.ops import resources

KERNELS = Path(__file__).parent.parent / "csrc" / "kernels"


def constants(source):
    """The whole numbers that a source names, where their expressions are made of such."""
    known = {}
    for names in re.findall(r"^constexpr int ([^;]+);", source, re.M):
        for part in names.split(", "):
            name, _, value = part.partition(" = ")
            value = re.sub(r"/\*.*?\*/", "", value)
            if re.fullmatch(r"[\w\s+*/()-]+", value or "."):
                try:
                    known[name.strip()] = int(eval(value.replace("/", "//"), {}, dict(known)))
                except (NameError, SyntaxError):
                    pass
    return known


@pytest.mark.parametrize("kernel,source,threads,smem", [
    ("gemm_bf16_kernel", "gemm_sm100.cu", "THREADS", "SMEM_BYTES"), ("gemm_pair_kernel", "gemm_pair_sm100.cu", "THREADS", "SMEM_BYTES"),
    ("gemm_mx_kernel", "gemm_mx_sm100.cu", "THREADS", "SMEM_BYTES"), ("flash_fwd_kernel", "flash_fwd_sm100.cu", "THREADS", None),
    ("flash_fwd_pair_kernel", "flash_fwd_pair_sm100.cu", "THREADS", None), ("flash_dq_kernel", "flash_bwd_sm100.cu", "THREADS", None),
    ("flash_dkv_kernel", "flash_bwd_sm100.cu", "THREADS", None)])
def test_launch_shapes(kernel, source, threads, smem):
    known, launch = constants((KERNELS / source).read_text()), resources.LAUNCHES[kernel]
    assert launch.threads == known[threads]
    assert smem is None or launch.dynamic_smem == known[smem]
