"""The schedule of the plain form's line sweeps on a cluster (k_wsor and
plain_sor of trans_bl_gb300/csrc/tb_plain.cu) restated in Python and checked
against the reference's sequential order (sor, poisson_par.f:167-226) on a
model problem: each line update is a nonlinear function of the lines its
stencil reads, so any value from the wrong sweep changes the result.

A slot runs the sweeps q, q + NS, ... on a ring of 16 lines (two rings in
turn where it runs several), the first sweep is fed from the field, every
sweep hands its lines on to the slot behind it, the far border line ahead of
the others, and the last sweep writes them back.  Within a step nothing is
ordered: no task may read what another one writes.
"""
import numpy as np
import pytest

LAG, RING = 5, 16


def update(line, m, F):
    """New value of a line from the lines its stencil reads (model of one line solve)."""
    if line == 1:
        nb = (0, 2, 3, 4, 5)
    elif line == m:
        nb = (m + 1, m - 1, m - 2, m - 3, m - 4)
    else:
        nb = (line - 2, line - 1, line + 1, line + 2)
    w = (0.31, 0.17, 0.23, 0.11, 0.07)
    return np.sin(F(line) + sum(a * F(q) for a, q in zip(w, nb))) + 0.01 * line, nb + (line,)


def sequential(F, ns):
    F = F.copy()
    m = F.shape[0] - 2
    for _ in range(ns):
        for line in [1, m] + list(range(2, m)):
            F[line] = update(line, m, lambda q: F[q])[0]
    return F


def sweeps(F, ns, C, W, parity):
    """One launch: `ns` sweeps on C CTAs of W slots with `parity` rings each, in place."""
    nxl = F.shape[0]
    m, NS = nxl - 2, C * W
    rings = [[dict() for _ in range(parity)] for _ in range(NS)]   # cell -> (line, sweep it comes from, value)

    def ring(s):
        return rings[s % NS][(s // NS) & 1 if parity > 1 else 0]

    for q in range(1, min(m, 7) + 1):
        ring(0)[q % RING] = (q, -1, F[q].copy())
    edge = {0: F[0].copy(), nxl - 1: F[nxl - 1].copy()}
    turn = LAG * NS if parity > 1 else 1 << 30
    current = list(range(NS))            # the sweep a slot's line group is at
    border = [W * r for r in range(C)]   # that of the first slot a CTA's border group watches

    for t in range(m - 1 + LAG * (ns - 1)):
        tasks = []
        for sw in current:
            s = sw + (NS if t - LAG * sw >= turn else 0)
            u = t - LAG * s
            if 0 <= u <= m - 2 and s < ns:
                tasks.append((s, u + 1))
        for sw in border:
            for q in range(W):
                s = sw + q
                s += NS if t - LAG * s >= turn else 0
                if t - LAG * s == m - 6 and s < ns:
                    tasks.append((s, m))
                    break
        reads, writes = set(), []
        for s, line in tasks:
            R = ring(s)

            def value(q, R=R, s=s):
                if q in edge:
                    return edge[q]
                got = R[q % RING]
                assert got[0] == q, "sweep %d step %d: the ring holds line %d for %d" % (s, t, got[0], q)
                return got[2]

            new, touched = update(line, m, value)
            reads |= {(id(R), q % RING) for q in touched if q not in edge and q != line}
            writes.append((R, line, s, new))
            if s + 1 < ns:
                writes.append((ring(s + 1), line, s, new))
        if t + 8 <= m:
            writes.append((ring(0), t + 8, -1, F[t + 8].copy()))
        cells = [(id(R), line % RING) for R, line, _, _ in writes]
        assert len(set(cells)) == len(cells), "two writes of one cell at step %d" % t
        assert not set(cells) & reads, "a cell read by a task is written by another at step %d" % t
        for R, line, s, v in writes:
            R[line % RING] = (line, s, v)
        for s, line in tasks:
            if s == ns - 1:
                F[line] = ring(s)[line % RING][2]
        current = [sw + (NS if t + 1 - LAG * sw >= turn else 0) for sw in current]
        border = [sw + (NS if t + 1 - LAG * sw - LAG * (W - 1) >= turn else 0) for sw in border]


def launches(nxl, itera, warps):
    """plain_sor's cut of `itera` sweeps into launches: sweeps, CTAs, slots of a
    CTA (up to three where a line takes one warp), rings."""
    m = nxl - 2
    done = 0
    while done < itera:
        ns, C, W, parity = itera - done, 1, 1, 1
        want = min(ns, (m - 1 + LAG - 1) // LAG)
        most = 3 if warps == 1 else 1
        if want > 1:
            if want > most:
                C = 2
                while C < 8 and C * most < want:
                    C *= 2
            W = min(most, (want + C - 1) // C)
        if ns > C * W:
            if m - 1 <= LAG * C * W:
                parity = 2
            else:
                ns = C * W
        yield ns, C, W, parity
        done += ns


@pytest.mark.parametrize("nxl", [9, 10, 13, 17, 22, 23, 27, 28, 33, 49, 65, 97, 121, 129])
@pytest.mark.parametrize("itera", [1, 2, 3, 4, 60])
@pytest.mark.parametrize("warps", [1, 4])
def test_sweeps_equal_sequential(nxl, itera, warps):
    F = np.random.default_rng(nxl * 100 + itera).standard_normal((nxl, 5))
    ref = sequential(F, itera)
    for ns, C, W, parity in launches(nxl, itera, warps):
        sweeps(F, ns, C, W, parity)
    np.testing.assert_array_equal(F, ref)
