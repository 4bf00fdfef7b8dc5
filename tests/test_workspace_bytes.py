"""workspace_bytes covers the partial sums of the coherent sum that image() runs, in every form, packed or not (no GPU)."""
import random

import torch

from opticalimaging_b200 import engine as E


def _model(z, k, packed, b, ny, nx):
    m = object.__new__(E.CoherentModel)
    m.band, m.ny, m.nx, m.form = E.Band(-(b // 2), b, -(b // 2), b), ny, nx, None
    m.pupils = torch.empty((z, k, b, b), dtype=torch.complex64, device='meta')
    m.packed = (torch.empty((z, packed, b, b), dtype=torch.complex64, device='meta'), None) if packed else None
    p = m.plan = object.__new__(E.Plan)
    p.ny, p.nx, p.band, p.mr, p.mc = ny, nx, m.band, E.coarse_size(b), E.coarse_size(b)
    p.coarse_fft, p.coarse256 = p.mr in (64, 128), p.mr == 256
    return m


def test_partial_sums_fit():
    rng = random.Random(7)
    for _ in range(3000):
        k = int(2 ** rng.uniform(0, 9))
        packed = rng.choice((0, 0, (k + 1) // 2, rng.randint(1, k)))
        z, batch, nch = rng.choice((1, 1, 3)), int(2 ** rng.uniform(0, 7)), rng.choice((1, 1, 3))
        m = _model(z, k, packed, rng.choice((9, 31, 59, 90, 117)), 300, 280)
        for form in (None, 'fft', 'dft'):
            for n in {k, packed if packed and nch == 1 else k}:
                p = m.plan
                if form != 'dft' and (p.coarse_fft or p.coarse256):
                    parts = E.field_split_sm(n * nch, batch * z)
                else:
                    parts = E.field_split(n * nch, batch * z * ((p.mr + 15) // 16))
                assert m.workspace_bytes(batch, nch, form) >= 4 * parts * batch * z * p.mr * p.mc
