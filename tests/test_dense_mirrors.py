"""The structures that csrc/dense_layer.cu and kernels/dense.py share, field by field (no GPU)."""
from __future__ import annotations

import ctypes as C
import re

import pytest

from inference_bench_b200.kernels import build, dense

TYPES = {"int": C.c_int, "float": C.c_float, "long long": C.c_longlong, "IbDenseProduct": dense.Product, "cudaStream_t": C.c_void_p}


def _fields(name: str) -> list:
    """[(field, ctypes type)] of a structure in the source; a pointer stands in a declaration of its own."""
    text = re.sub(r"//[^\n]*", "", (build.CSRC / "dense_layer.cu").read_text())
    body = re.search(r"struct %s \{(.*?)\n\};" % name, text, re.S).group(1)
    out = []
    for decl in filter(None, (" ".join(d.split()) for d in body.split(";"))):
        pointer = re.fullmatch(r"(?:const )?\w+\* (\w+)", decl)
        if pointer:
            out.append((pointer.group(1), C.c_void_p))
            continue
        kind, names = re.fullmatch(r"(long long|\w+) ([\w, ]+)", decl).groups()
        out += [(n.strip(), TYPES[kind]) for n in names.split(",")]
    return out


@pytest.mark.parametrize("name,mirror", [("IbDenseProduct", dense.Product), ("IbDenseStep", dense.DenseStep), ("IbDenseLayer", dense.DenseLayer)])
def test_fields(name, mirror):
    assert _fields(name) == list(mirror._fields_)


def test_sizes():
    dense._check_mirrors()
