"""What an installed package holds: everything the kernel library and the extension over it are made of, and both objects."""
import tomllib
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
PKG = ROOT / "maxdiffusion_b200"


def test_the_package_holds_sources_and_objects():
  patterns = tomllib.loads((ROOT / "pyproject.toml").read_text())["tool"]["setuptools"]["package-data"]["maxdiffusion_b200"]
  files = {p.relative_to(PKG).as_posix() for pattern in patterns for p in PKG.glob(pattern)}
  sources = {f"csrc/{p.name}" for p in (PKG / "csrc").iterdir() if p.suffix in (".cu", ".cuh", ".h", ".cpp")}
  assert "csrc/host_ops.cpp" in sources and sources <= files, sources - files
  assert {"_kernels.so", "_host_ops.so"} <= set(patterns)
