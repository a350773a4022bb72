"""Saved state and loading: what a restore must refuse before the context
changes, and a context whose filaments could not be loaded."""
import struct

import numpy as np
import pytest

from test_gpu_parity import _payload_hash

pytestmark = pytest.mark.gpu


def _entry_regions(ctx, blob):
    """Offsets of the entry ranges e_off and e_cnt in a one-system checkpoint:
    after the capacity, 13 site arrays of doubles, two filament int arrays, the
    displacement maximum, the pair count (int) and the rebuild counter."""
    at = 96 + 4 + 13 * 8 * ctx.n_sites + 8 * ctx.n_fil + 8 + 4 + 8
    return at, at + 4 * (ctx.n_sites - ctx.n_fil)


def test_restore_rejects_entries_apart():
    """Bonds' entry ranges that each lie inside their segment, but not one
    after the other, are refused: a lane of the team integrator reads its two
    bonds' slots as one run.  (The first bond's empty range is moved to the
    segment's end, its neighbour's keeps its entries.)"""
    import simcore_b200 as sc
    from simcore_b200 import workloads
    cfg = workloads.make("B", scale=0.02, seed=5)
    a, b = (sc.Context(*cfg[:3], precision="fp64") for _ in range(2))
    a.step(5)
    b.step(5)
    blob = bytearray(a.checkpoint())
    e_off, e_cnt = _entry_regions(a, blob)
    n_bonds = a.n_sites - a.n_fil
    off = np.frombuffer(blob, "<i4", n_bonds, e_off)
    cnt = np.frombuffer(blob, "<i4", n_bonds, e_cnt)
    assert np.array_equal(off[1:], off[:-1] + cnt[:-1])  # the library's own lists
    cap = struct.unpack_from("<i", blob, 96)[0]
    per = n_bonds // a.n_fil
    first = next(i for i in range(n_bonds)
                 if i % per != per - 1 and cnt[i] == 0 and cnt[i + 1] > 0)
    bad = bytearray(blob)
    struct.pack_into("<i", bad, e_off + 4 * first, 2 * cap)
    struct.pack_into("<Q", bad, 88, _payload_hash(bytes(bad[96:])))
    with pytest.raises(sc.ScError, match="apart"):
        a.restore(bytes(bad))
    a.step(4)
    b.step(4)
    assert np.array_equal(a.sites(), b.sites())
    a.restore(bytes(blob))
    b.restore(bytes(blob))
    a.step(4)
    b.step_graph(4)
    assert np.array_equal(a.sites(), b.sites())
    a.close()
    b.close()
