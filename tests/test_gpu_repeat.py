"""Batched solves of the common kernel repeat bit for bit: every sum of an SCF runs in a fixed order, whichever CTA takes the job,
wherever its matrices lie and whatever else is in the launch. (Gradients are added by atomics and repeat to rounding; solves under
second-derivative tolerances add atomically too.)"""
import numpy as np
import pytest

from helpers import A2B
from pm3_rs import _lib, native, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("multiplicity,grow", [(1, workloads.organic), (2, workloads.radical)])
def test_solves_repeat_bit_for_bit(multiplicity, grow):
    mols = [grow(n, 40 + n) for n in (6, 9, 14, 23, 31, 40)]
    beside = [workloads.water_cluster(42, grid=(4, 4, 3))] if multiplicity == 1 else [grow(52, 3)]
    opts = native.options(multiplicity=multiplicity, max_scf=1000)
    runs = []
    for batch in (mols, mols, mols[::-1], mols + beside):
        offs, z, xyz = workloads.pack(batch)
        c = _lib.Context()
        try:
            r = native.batch(offs, z, xyz * A2B, opts, context=c)
        finally:
            c.close()
        order = list(range(len(mols)))
        if batch[0] is mols[-1]:
            order.reverse()
        runs.append((r.status[order], r.iterations[order], r.electronic_ev[order], r.homo_ev[order],
                     np.concatenate([r.charges_of(m) for m in order])))
    for other in runs[1:]:
        for a, b in zip(runs[0], other):
            assert np.array_equal(a, b)
