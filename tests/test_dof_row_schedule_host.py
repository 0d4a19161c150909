"""The row schedule that follows the entry schedule in ``br_dof_schedule``'s output, which the LM kernel
runs: interpreted on the CPU exactly as the kernel reads it, it must do the entry schedule's operations
entry by entry in the same order (equal to the last bit in float32 and float64), keep every access inside
its rows, and write every entry of a level from one task; the trunk's rows take the levels' contributions
in one sweep, in their order."""

import numpy as np
import pytest

from test_dof_schedule_host import _contribs, _decode, _dof_parents, _random_tree_matrix, _schedule, _tree, _trunk


def _rows(s):
    nlev, ntask, nextra = (int(v) for v in s[:3])
    roff = (((5 + nlev + 3) & ~3) + 4 * ntask + 2 * nextra + 3) & ~3
    n, nx, lv, nr = (int(v) for v in s[roff:roff + 4])
    levels, ntr = lv & 0xffff, lv >> 16
    assert levels + ntr == nlev
    t = roff + ((5 + nlev + 3) & ~3)
    trunk = s[t + 4 * n + nx:].astype(np.int64)
    return s[roff + 4:roff + 5 + levels].astype(np.int64), s[t:t + 4 * n].reshape(n, 4).astype(np.int64), \
        s[t + 4 * n:t + 4 * n + nx].astype(np.int64), nr, ntr, trunk


def _trees():
    out = dict(_dof_parents())
    out["chain62"] = np.arange(-1, 61, dtype=np.int32)
    out["binary64"] = np.array([-1] + [(c - 1) // 2 for c in range(1, 64)], np.int32)
    for seed in range(6):
        rng = np.random.default_rng(seed)
        n = int(rng.integers(1, 65))
        out[f"random{seed}"] = np.array([int(rng.integers(-1, c)) for c in range(n)], np.int32)
    return out


@pytest.mark.parametrize("name", sorted(_trees()))
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_row_schedule_equals_entry_schedule(name, dtype):
    dp = _trees()[name]
    nv, s = len(dp), _schedule(dp)
    dep, anc, rowoff = _tree(dp)
    ro = np.cumsum([0] + [(d + 3) & ~1 for d in dep])
    starts, tasks, extra, nr, ntr, trunk = _rows(s)
    assert ntr == _trunk(dp) and len(trunk) == (nv - ntr if ntr else 0)
    assert nr == ro[-1]
    owner = np.repeat(np.arange(nv), np.diff(ro))
    rng = np.random.default_rng(nv)
    A, g = _random_tree_matrix(dp, rng).astype(dtype), rng.normal(size=nv).astype(dtype)
    damp, zoff = dtype(1e-2), rowoff[nv]
    m = np.zeros(zoff + nv, dtype)                      # the entry schedule's storage
    r = np.full(nr, np.nan, dtype)                      # the row schedule's; padding is never used
    at = np.zeros(zoff + nv, np.int64)                  # where an entry of the first lies in the second
    for c in range(nv):
        for b, p in enumerate(anc[c] + [c]):
            m[rowoff[c] + b], at[rowoff[c] + b] = A[c, p], ro[c] + 1 + b
        m[zoff + c], at[zoff + c] = -g[c], ro[c]
    r[at] = m
    r[np.isnan(r)] = 0.0
    dinv = np.array([dtype(1) / (m[rowoff[c] + dep[c]] + damp) for c in range(nv)])
    dinv_r = dinv.copy()
    nlev, _, estarts, etasks, eextra = _decode(s)
    for lev in range(nlev):
        for tk in etasks[estarts[lev]:estarts[lev + 1]]:
            d = tk[0] & 0xffff
            for a, b, k in _contribs(tk, eextra):
                m[d] = m[d] - (m[a] * dinv[k]) * m[b]
            if tk[3]:
                dinv[tk[3] - 1] = dtype(1) / (m[d] + damp)
        if lev >= nlev - ntr:                           # the trunk's own levels
            k = nlev - 1 - lev
            if k == ntr - 1:                            # every other DOF's contributions, in one sweep
                for w in trunk:
                    o, d = w & 0xffff, w >> 16
                    assert o == ro[d]
                    for i in range(ntr):
                        e = np.arange(i + 2)
                        r[ro[i] + e] = r[ro[i] + e] - (r[o + 1 + i] * dinv_r[d]) * r[o + e]
                dinv_r[k] = dtype(1) / (r[ro[k] + 1 + k] + damp)
            for i in range(k):
                e = np.arange(i + 2)
                r[ro[i] + e] = r[ro[i] + e] - (r[ro[k] + 1 + i] * dinv_r[k]) * r[ro[k] + e]
            if k > 0:
                dinv_r[k - 1] = dtype(1) / (r[ro[k - 1] + k] + damp)
            np.testing.assert_array_equal(r[at], m)
            np.testing.assert_array_equal(dinv_r, dinv)
            continue
        written, read = [], set()
        for x, c0, z, c1 in tasks[starts[lev]:starts[lev + 1]]:
            dst, delta, n = x & 0xffff, (x >> 16) & 0xff, x >> 24
            f, width = (z >> 16) & 0x7fff, 4 if z >> 31 else 2
            assert owner[dst] >= ntr and dst % 2 == 0 and len(set(owner[dst:dst + width])) == 1 and dst + width <= nr
            cs = [c0] + ([c1] if n > 1 else []) + list(extra[(z & 0xffff):(z & 0xffff) + max(0, n - 2)])
            assert len(cs) == n
            for c in cs:
                so, k = c & 0xffff, c >> 16
                src = so - delta
                assert src % 2 == 0 and set(owner[src:src + width]) == {k} and owner[so] == k
                assert anc[k][so - ro[k] - 1] == owner[dst]
                r[dst:dst + width] = r[dst:dst + width] - (r[so] * dinv_r[k]) * r[src:src + width]
                read.add(int(k))
            written += list(range(dst, dst + width))
            if f:
                assert dst + delta == ro[f - 1] + 1 + dep[f - 1]
                dinv_r[f - 1] = dtype(1) / (r[dst + delta] + damp)
        assert len(written) == len(set(written)) and not read & {int(owner[w]) for w in written}
        below = at if ntr == 0 else np.array([x for x in at if owner[x] >= ntr])
        np.testing.assert_array_equal(r[below], m[np.isin(at, below)])
        np.testing.assert_array_equal(dinv_r[ntr:], dinv[ntr:])
    x = np.zeros(nv)                                    # and it solves the system
    for c in sorted(range(nv), key=lambda c: dep[c]):
        x[c] = (r[ro[c]] - sum(float(r[ro[c] + 1 + a]) * x[p] for a, p in enumerate(anc[c]))) * dinv_r[c]
    ref = np.linalg.solve(A.astype(float) + float(damp) * np.eye(nv), -g.astype(float))
    tol = 1e-8 if dtype is np.float64 else 1e-4 * np.linalg.cond(A.astype(float) + float(damp) * np.eye(nv))
    assert np.abs(x - ref).max() <= tol * max(1.0, np.abs(ref).max())
