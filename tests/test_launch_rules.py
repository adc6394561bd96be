"""Rules of launches that overlap their predecessor (ani_launch.cuh) which no run can show to be kept: they are checked on
the source."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "khan_b200", "csrc")

# kernels that read the molecules ahead of their wait, and what the kernel in front of each may still be writing then
EARLY_READERS = [
    ("ani_featurize_mol.cuh", "featurize_mol_kernel", ["scatter"]),
    ("ani_featurize_mol.cuh", "load_sorted_molecule", ["scatter"]),
    ("ani_grad_mol.cuh", "featurize_grad_mol_kernel", ["gh", "gc", "gn", "go", "grow", "atom_energy_sorted"]),
]


def function(file, name):
    """(parameter list, body) of a function, without comments."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, file)).read())
    params, rest = re.search(r"\b%s\((.*?)\)\s*\{(.*)" % name, text, re.S).groups()
    return params, rest[:rest.index("\n}\n")]


@pytest.mark.parametrize("file,name,written", EARLY_READERS)
def test_what_the_kernel_in_front_writes_is_read_in_its_place(file, name, written):
    params, body = function(file, name)
    assert "pdl_wait" in body
    for array in written:
        assert not re.search(r"__restrict__\s+%s\b" % array, params), array
        assert not re.search(r"\b%s\s*\[" % array, body), array


def test_a_batch_without_molecules_to_work_on_waits_too():
    """All molecules without atoms: some CTA must wait all the same, or the kernel behind runs beside the one in front."""
    for file, name, failed in (("ani_featurize_mol.cuh", "featurize_mol_kernel", r"if \(!load_molecule\([^;{]*\)\)"),
                               ("ani_grad_mol.cuh", "featurize_grad_mol_kernel", r"if \(!usable\)")):
        assert re.search(failed + r" \{\s*pdl_wait\(\);", function(file, name)[1]), name
