"""Credit tables of custom groups against the lookup of one atom at a time."""
import numpy as np
import pytest


@pytest.mark.parametrize("kind", ["disjoint", "overlapping", "unsorted", "repeated"])
def test_credit_tables(cm, kind):
    rng = np.random.default_rng(7)
    atoms = list(range(11, 71))
    groups = [sorted(rng.choice(atoms, size=int(n), replace=False).tolist()) for n in rng.integers(1, 20, size=9)]
    if kind == "disjoint":
        groups = [atoms[i : i + 7] for i in range(0, 50, 7)]
    sel = cm.AtomSelection.from_indices(atoms, natomspermol=20, group_atom_indices=groups,
                                        group_names=[str(i) for i in range(len(groups))])
    if kind == "unsorted":
        sel.group_atom_indices[2] = [40, 12, 33, 15]
    if kind == "repeated":
        sel.group_atom_indices[1] = [12, 12, 40]
    assert sel.solute_credit_table() == [sel.groups_of_index(i) for i in atoms[:20]]
    assert sel.solvent_credit_table() == [sel.groups_of_index(i) for i in atoms]
