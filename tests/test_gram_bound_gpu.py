"""etm_count_tiles_tc_bound: the survivors, counts and bits of a host Gram, for block pairs that stop early, late or not
at all. Zero tolerance."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

T = 240


def _rows(rng, m, words, dens):
    """Member rows uint64 [m, words] with row i's bits set with probability dens[i]."""
    return np.stack([np.packbits(rng.random(words * 64) < d, bitorder="little").view(np.uint64) for d in dens])


@pytest.mark.parametrize("with_cls", [False, True])
@pytest.mark.parametrize("shape", ["ascending", "descending", "late", "clustered", "none", "all"])
def test_survivors_match_the_host(pkg, shape, with_cls):
    """Groups of one block (under and over half of it), of two and three, over stages short of a check and past it;
    members of ascending or descending support, pairs that meet only in the last rows, or in the first."""
    import torch

    lib = pkg.load_library()
    rng = np.random.default_rng(len(shape))
    sizes = np.array([100, 121, 240, 241, 500, 2, 300], np.int64)
    cw = np.array([400, 700, 128, 513, 260, 300, 60], np.int64)
    cld = (cw + 31) // 32 * 32
    alloc = -(-sizes // T) * T
    cbase = np.zeros(len(sizes), np.int64)
    cbase[1:] = np.cumsum(alloc * cld)[:-1]
    buf = rng.integers(-2**62, 2**62, int((alloc * cld).sum()), dtype=np.int64).view(np.uint64)  # past m: anything
    want, totals = [], []
    for g, (m, w) in enumerate(zip(sizes, cw)):
        dens = np.sort(rng.uniform(0.02, 0.25, m))
        if shape == "descending":
            dens = dens[::-1]
        x = _rows(rng, m, w, dens)
        if shape in ("late", "clustered"):
            # Two in five members share a run of rows near the end, or at the start.
            some = rng.random(m) < 0.4
            at = slice(w - w // 8, w) if shape == "late" else slice(0, w // 8)
            x[some, at] = 2**64 - 1
        full = np.zeros((m, cld[g]), np.uint64)
        full[:, :w] = x
        j, ww = np.arange(m)[:, None], np.arange(cld[g])[None, :]
        buf[cbase[g] + (j // T) * cld[g] * T + (ww // 4) * 4 * T + (ww // 2 % 2) * 2 * T + (j % T) * 2 + ww % 2] = full
        bits = np.unpackbits(x.view(np.uint8), axis=1).astype(np.float32)
        gram = (bits @ bits.T).astype(np.int64)
        want.append(gram[np.triu_indices(m, 1)])
        totals.append(np.diagonal(gram))
    want = np.concatenate(want)
    mc = {"none": 10**6, "all": 1}.get(shape, int(np.quantile(want, 0.97)))
    cand_off = np.zeros(len(sizes) + 1, np.int64)
    np.cumsum(sizes * (sizes - 1) // 2, out=cand_off[1:])
    nb = alloc // T
    work_off = np.zeros(len(sizes) + 1, np.int64)
    np.cumsum(nb * (nb + 1) // 2, out=work_off[1:])
    first = np.cumsum(sizes) - sizes + 3  # the groups' rows start at row 3 of the level
    counts = np.concatenate([[7, 7, 7], *totals]).astype(np.int32)
    cls = rng.integers(0, 3, len(want)).astype(np.uint8)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (
        buf.view(np.int64), cbase, cw, cld, sizes.astype(np.int32), cand_off, np.arange(len(sizes)), work_off, first,
        counts, cls)]
    out = torch.full((len(want),), -1, dtype=torch.int32, device="cuda")
    bits = torch.zeros(len(want) // 32 + 2, dtype=torch.int32, device="cuda")
    counter = torch.zeros(1, dtype=torch.int64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    st = lib.etm_count_tiles_tc_bound(*(x.data_ptr() for x in d[:8]), len(sizes), int(work_off[-1]), 0,
                                      d[10].data_ptr() if with_cls else None, mc, out.data_ptr(), bits.data_ptr(),
                                      d[8].data_ptr(), d[9].data_ptr(), counter.data_ptr(), stream)
    assert st == 0, lib.etm_last_error()
    assert lib.etm_device_status(stream) == 0
    keep = want >= mc
    if with_cls:
        keep &= cls == 0
    assert np.array_equal(out.cpu().numpy(), np.where(keep, want, -1))
    got = np.unpackbits(bits.cpu().numpy().view(np.uint8), bitorder="little")[:len(want)].astype(bool)
    assert np.array_equal(got, keep)
