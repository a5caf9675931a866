"""GPU tests of the host path: pooled streams and blocks under threads, and host tensors around the
sizes where the staging changes (one thread and one slab, several slabs, slabs with a remainder)."""
import threading

import numpy as np
import pytest

from gbasis_b200 import _engine
from gbasis_b200 import electron_repulsion as er
from gbasis_b200.batch import electron_repulsion_integral_batch
from gbasis_b200.synthetic import batch_molecule, make_workload, random_shell

pytestmark = pytest.mark.gpu


def _molecule(n_functions):
    """s and p shells with n_functions Cartesian functions."""
    rng = np.random.default_rng(n_functions)
    n_p = n_functions // 6
    ls = [1] * n_p + [0] * (n_functions - 3 * n_p)
    return [random_shell(rng, l, 1, rng.uniform(0.0, 4.0, 3)) for l in ls]


@pytest.mark.parametrize("n", [1, 2, 22, 23, 24, 37, 46])
def test_host_tensor_sizes(n):
    """The streamed host tensor equals the device tensor at every staging size (2 MB is n = 22.6;
    37 and 46 leave a remainder in the last slab)."""
    import torch
    db = _engine.DeviceBasis(_molecule(n))
    assert db.nbf == n
    dev = torch.empty((n,) * 4, dtype=torch.float64, device="cuda")
    for notation in ("chemist", "physicist"):
        db.full_device(dev.data_ptr(), notation)
        torch.cuda.synchronize()
        ref = dev.cpu().numpy()
        np.testing.assert_array_equal(db.full_host(notation), ref)
        pinned = torch.empty((n,) * 4, dtype=torch.float64, pin_memory=True).numpy()
        np.testing.assert_array_equal(db.full_host(notation, out=pinned), ref)
    db.close()


def test_threads_share_the_pools():
    """More threads than pooled stream sets, each with its own molecules, batches among them, while
    the pools are emptied: every result is the serial one, bit for bit."""
    mols = [make_workload("tiny4")] + [batch_molecule(m) for m in (3, 8, 21)]
    ref = [er.electron_repulsion_integral(m) for m in mols]
    ref_b = [t.cpu().numpy() for t in electron_repulsion_integral_batch(mols[:2])]
    errors = []

    def work(k):
        try:
            for rep in range(6):
                m = (k + rep) % len(mols)
                np.testing.assert_array_equal(er.electron_repulsion_integral(mols[m]), ref[m])
                if rep % 3 == 0:
                    for t, r in zip(electron_repulsion_integral_batch(mols[:2]), ref_b):
                        np.testing.assert_array_equal(t.cpu().numpy(), r)
                if k == 0:
                    _engine.release_cached_memory()
        except BaseException as e:  # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(7)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
