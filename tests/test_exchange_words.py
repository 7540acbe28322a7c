"""Kernels that exchange data without fences poll words that carry their own
sequence number, so each (value, number) pair has to be read and written whole.
PTX gives a vector access no more than the single accesses of its elements, in
any order: a pair of 32-bit halves is whole as one 64-bit element and not as two
32-bit ones. Checked on the source; a torn pair cannot be provoked in a run."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "apc_524_project_gb300", "csrc")
VECTOR = re.compile(r'"\s*(?:ld|st)\.(?:volatile|relaxed|acquire|release)[\w.:]*\.v[248]\.[a-z](\d+)')


def _vector_accesses():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                for bits in VECTOR.findall(f.read()):
                    yield name, int(bits)


def test_polled_pairs_are_single_elements():
    found = list(_vector_accesses())
    assert {name for name, _ in found} == {"fields_f64.cu"} and len(found) == 2  # the Jacobi tiles' send and receive
    assert all(bits == 64 for _, bits in found), found
