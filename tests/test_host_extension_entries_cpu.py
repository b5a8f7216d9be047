"""The entry points that the host extension calls: their declarations are the kernel library's definitions, and those that it
needs have the arguments that every library with them has (a change of arguments takes another name)."""
import re

from maxdiffusion_b200 import build

_SIGNATURE = r"\bint (mdb_\w+)\(([^)]*)\)\s*"


def _types(params):
  params = re.sub(r"\bMdb\w+", "void", params)  # a structure is passed as an address
  return [re.sub(r"\s*\b(?!const\b|void\b|int\b|float\b|long\b|unsigned\b)[A-Za-z_]\w*\s*$", "", " ".join(p.split())).replace(" *", "*") for p in params.split(",")]


def test_declarations_are_the_definitions():
  host = (build.SRC_DIR / "host_ops.cpp").read_text()
  declared = dict(re.findall(_SIGNATURE + ";", host))
  defined = {}
  for src in build.sources():
    text = src.read_text()
    if src.name == "flash_fwd.cu":  # generated per head size
      text += text.replace("##SUFFIX", "").replace("\\\n", "\n") + text.replace("##SUFFIX", "_d64").replace("\\\n", "\n")
    defined.update(re.findall(_SIGNATURE + r"\{", re.sub(r"//[^\n]*", "", text)))
  assert len(declared) >= 12
  for name, params in declared.items():
    assert name in defined and _types(params) == _types(defined[name]), name
  assert len(declared["mdb_gn_cl_fold_fwd"].split(",")) == 15
