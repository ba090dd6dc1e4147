"""CPU check of what bench.py calls the dominant kernel: one of the main chain,
with its committed DRAM bytes and instruction count."""
import importlib.util
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_dominant_kernel_is_on_the_main_chain():
    spec = importlib.util.spec_from_file_location("bench", ROOT / "bench.py")
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    share = {"solid_solve": 0.21, "density": 0.19, "xsph": 0.15, "contact_mark": 0.3, "scan": 0.03}
    dom = bench.dominant_kernel({k: {"share": v} for k, v in share.items()})
    assert dom == "density"
    assert bench.ncu_traffic(dom, "gpu_default") and bench.ncu_instructions(dom, "gpu_default")
