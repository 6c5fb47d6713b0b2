"""A run with an op that the engine refuses behind measurements that the device decides: the
call fails, and what came before the op has happened, its draws from the generator too."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _refused(n):
    # a phase polynomial of 513 terms: the dense kernel takes 512
    terms = ";".join(f"{1 + k % 7}:{1 << (k % n)}" for k in range(513))
    return f"DIAG(3;0;{terms}) {' '.join(map(str, range(n)))}"


@pytest.mark.parametrize("n,precision,measured", [(11, 0, 2), (13, 1, 5), (11, 0, 300)])
def test_the_draws_before_a_refused_op_are_taken(n, precision, measured):
    import ncsim_b200 as nb

    before = []
    for k in range(measured):  # each outcome uncertain: one draw
        before += [f"H {k % n}", f"M {k % n}"]
    head = f"QUBITS {n}\n" + "\n".join(before) + "\n"
    a, ra = nb.GpuStateVector(n, precision), nb.StdRng(measured)
    with pytest.raises(nb.SimError, match="512 terms"):
        a.run(nb.Circuit.parse(head + _refused(n) + "\nH 0\nM 0\n"), ra)
    b, rb = nb.GpuStateVector(n, precision), nb.StdRng(measured)
    b.run(nb.Circuit.parse(head), rb)
    assert np.array_equal(a.to_vector(), b.to_vector())
    last = ra.next_u64()
    assert last == rb.next_u64()
    rc = nb.StdRng(measured)
    for _ in range(measured):
        rc.gen_f64()
    assert last == rc.next_u64()
    # the register takes the next run
    more = nb.Circuit.parse(f"QUBITS {n}\nH 1\nM 1\n")
    assert a.run(more, ra) == b.run(more, rb)
