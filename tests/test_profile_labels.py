"""CPU check that the profile harness names every kernel of the library: instances of the GEMM template as the profiler and ncu
print them, and every ``__global__`` function of the sources."""
import itertools
import re
from pathlib import Path

from streamep_b200.stream_moe.profile_pipeline import GEMMS, KERNELS, classify
from streamep_b200.utils.roofline import Peaks, layer_rooflines, single_rank_rooflines

CSRC = Path(__file__).resolve().parent.parent / "streamep_b200" / "csrc"


def test_every_kernel_of_the_sources_has_a_name():
    found = set()
    for f in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        found |= set(re.findall(r"__global__\s+void\b[^{;]*?(\w+_kernel)\s*\(", text, re.S))
    assert found == set(KERNELS) | {"grouped_gemm_kernel"}
    for name in KERNELS:
        for form in (f"sep::{name}(sep::Params)", f"void sep::{name}<1>(sep::Params)", f"void sep::{name}<(int)4, (int)64>(Params)"):
            assert classify(form) == KERNELS[name]


def test_every_gemm_instance_has_a_name():
    for (a, b, epi, push), label in GEMMS.items():
        for bn, cg in itertools.product((128, 256), (1, 2)):
            t = ("false", "true")
            forms = (f"{bn}, {t[a]}, {t[b]}, {epi}, {t[push]}, {cg}", f"{bn}, {a}, {b}, {epi}, {push}, {cg}",
                     f"(int){bn}, (bool){a}, (bool){b}, (int){epi}, (bool){push}, (int){cg}")
            for f in forms:
                assert classify(f"void sep::grouped_gemm_kernel<{f}>(CUtensorMap, CUtensorMap, sep::GemmParams)") == label
    assert classify("void at::native::vectorized_elementwise_kernel<4, at::native::FillFunctor<int>>(int)").startswith("memset")
    assert classify("ampere_gemm").startswith("other: ")


def test_rooflines_carry_the_names_of_the_kernels():
    labels = set(KERNELS.values()) | set(GEMMS.values())
    pk = Peaks(1400.0, 6500.0, 770.0, "test")
    fused, alone = layer_rooflines(8192, 2048, 1408, 6, 1, pk), single_rank_rooflines(8192, 2048, 1408, 6, pk)
    assert set(fused) | set(alone) <= labels and not set(fused) & set(alone)
    for a, b in (("GEMM-A SwiGLU", "dispatch (+) GEMM-A SwiGLU (fused)"), ("GEMM-Y_bwd dSwiGLU", "dispatch_grads (+) GEMM-Y_bwd dSwiGLU (fused)")):
        assert alone[a].flops == fused[b].flops and fused[b].hbm_bytes - alone[a].hbm_bytes == 2 * 8192 * 6 * 2048 * 2
