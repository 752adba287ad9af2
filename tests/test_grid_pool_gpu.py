"""Fields set up one after another and from several threads share the set-up's
memory pool and FFT plans: more sizes than plans are kept, revisited, and
concurrent set-ups on streams of their own give the planes of the first pass bit
for bit."""
import threading

import numpy as np
import pytest

from obit_b200.comps import CCField, CCModel
from obit_b200.grid import GridField, GridImage

pytestmark = pytest.mark.gpu


def _plane(n, stream=0):
    r = np.random.default_rng(n)
    cell = 1.0 / 3600.0
    ix, iy = r.integers(-n // 4, n // 4, (2, 200))
    field = CCField(flux=r.uniform(0.1, 1.0, 200).astype(np.float32), deltaX=(ix * -cell).astype(np.float32),
                    deltaY=(iy * cell).astype(np.float32), crvalRA=0.0, crvalDec=34.0, do3D=False, cdeltX=-cell,
                    cdeltY=cell)
    with GridField(field, GridImage(n, n, n / 2 + 1, n / 2 + 1), CCModel(uvRA=0.0, uvDec=34.0), stream=stream) as f:
        return f.plane()


def test_sizes_revisited_and_threads():
    torch = pytest.importorskip("torch")
    sizes = [64, 96, 128, 160, 192, 256]
    first = {n: _plane(n) for n in sizes}
    for n in sizes[::-1]:
        assert np.array_equal(_plane(n), first[n])
    bad = []

    def work(k):
        torch.cuda.set_device(0)
        st = torch.cuda.Stream()
        for n in sizes[k:] + sizes[:k]:
            if not np.array_equal(_plane(n, st.cuda_stream), first[n]):
                bad.append((k, n))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
