"""The resident solves' tiling (csrc/tse_resident.cuh) on the CPU: a restatement of its
address arithmetic.  Every cell belongs to one tile, every shared-memory index a sweep
touches lies inside the padded arrays, every edge word a tile reads is one its neighbour
writes, and the plans stay inside the blocks, cells and shared memory they are given."""
import random

import pytest

# floats or doubles a 16-byte group, most groups a tile and colour
FORMS = {"fp32": (4, 2 * 384), "fp64": (2, 65535)}


def plan(nx, ny, nz, vals, maxb, max_groups, smem_max, smem, threads):
    H = (nz + (nz & 1)) // 2
    Hg = -(-H // vals)
    best, cost0 = None, 0.0
    for gx0 in range(1, min(nx, maxb) + 1):
        ti = -(-nx // gx0)
        gx = -(-nx // ti)
        cap = maxb // gx
        for one in (0, 1):
            gyt = 1 if one else min(ny, cap)
            tj = -(-ny // gyt)
            gy = -(-ny // tj)
            pad = (ti + 2) * (tj + 2) * Hg + 2
            groups = ti * tj * Hg
            if groups > max_groups or pad > 65535 or ti > 250:
                continue
            halo = ((2 * tj if gx > 1 else 0) + (2 * ti if gy > 1 else 0)) * Hg
            P = dict(gx=gx, gy=gy, nb=gx * gy, ti=ti, tj=tj, pitch=tj + 2, pad=pad, halo=halo, Hg=Hg,
                     groups=groups)
            P["smem"] = smem(P)
            if P["smem"] > smem_max:
                continue
            cost = -1.0 if P["nb"] == 1 else groups + 0.5 * halo + (250.0 if halo > threads(P) else 0.0)
            if best is None or cost < cost0:
                best, cost0 = P, cost
    return best


def dc_smem(P):
    return 2 * P["pad"] * 16 + ((P["halo"] * 6 + 15) & ~15)


class Tile:
    def __init__(self, nx, ny, P, b):
        self.nx, self.ny, self.Hg, self.pitch = nx, ny, P["Hg"], P["pitch"]
        bi, bj = divmod(b, P["gy"])
        self.i0, i1 = bi * nx // P["gx"], (bi + 1) * nx // P["gx"]
        self.j0, j1 = bj * ny // P["gy"], (bj + 1) * ny // P["gy"]
        self.ti, self.tj = i1 - self.i0, j1 - self.j0
        self.groups = self.ti * self.tj * self.Hg

    def decode(self, u):
        o, g = divmod(u, self.Hg)
        if o < self.tj:
            return 0, o, g
        o -= self.tj
        if o < self.tj:
            return self.ti - 1, o, g
        o -= self.tj
        mid = self.ti - 2
        if o < mid:
            return 1 + o, 0, g
        o -= mid
        if o < mid:
            return 1 + o, self.tj - 1, g
        o -= mid
        a, b = divmod(o, self.tj - 2)
        return 1 + a, 1 + b, g

    def column(self, ci, cj):
        return (self.i0 + ci) * self.ny + self.j0 + cj

    def p(self, ci, cj, g):
        return ((ci + 1) * self.pitch + cj + 1) * self.Hg + g + 1

    def halos(self):
        """The kernel's numbering of the edge groups, word for word."""
        row, col = self.tj * self.Hg, self.ti * self.Hg
        n = (row if self.i0 > 0 else 0) + (row if self.i0 + self.ti < self.nx else 0)
        n += (col if self.j0 > 0 else 0) + (col if self.j0 + self.tj < self.ny else 0)
        return [self.halo(h, row, col) for h in range(n)]

    def halo(self, h, row, col):
        if self.i0 > 0:
            if h < row:
                return self.column(-1, 0) * self.Hg + h, self.p(-1, 0, h)
            h -= row
        if self.i0 + self.ti < self.nx:
            if h < row:
                return self.column(self.ti, 0) * self.Hg + h, self.p(self.ti, 0, h)
            h -= row
        cj = -1
        if self.j0 == 0 or h >= col:
            if self.j0 > 0:
                h -= col
            cj = self.tj
        ci, g = divmod(h, self.Hg)
        return self.column(ci, cj) * self.Hg + g, self.p(ci, cj, g)

    def shared(self, ci, cj):
        return ((ci == 0 and self.i0 > 0) or (ci == self.ti - 1 and self.i0 + self.ti < self.nx)
                or (cj == 0 and self.j0 > 0) or (cj == self.tj - 1 and self.j0 + self.tj < self.ny))


def _shapes():
    rng = random.Random(4)
    fixed = [(1, 1, 1), (1, 1, 40), (40, 1, 1), (5, 7, 2), (60, 1, 30), (16, 16, 16), (33, 17, 21),
             (1, 90, 7), (2, 2, 600), (3, 300, 4), (150, 2, 9)]
    return fixed + [tuple(rng.randint(1, 60) for _ in range(3)) for _ in range(25)]


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("maxb", [1, 7, 148])
def test_tiles_cover_the_grid_and_their_records_match(form, maxb):
    vals, max_groups = FORMS[form]
    planned = 0
    for nx, ny, nz in _shapes():
        P = plan(nx, ny, nz, vals, maxb, max_groups, 225 * 1024, SMEM[form], NTHREADS[form])
        if P is None:
            continue
        planned += 1
        assert P["nb"] <= maxb and P["smem"] <= 225 * 1024
        Hg, records = P["Hg"], nx * ny * P["Hg"]
        owner, published, wanted = {}, set(), set()
        for b in range(P["nb"]):
            T = Tile(nx, ny, P, b)
            assert 1 <= T.ti <= P["ti"] and 1 <= T.tj <= P["tj"] and T.groups <= P["groups"]
            rrow = (ny - T.pitch) * Hg
            rbase = T.column(0, 0) * Hg - (T.pitch + 1) * Hg - 1
            places = set()
            for u in range(T.groups):
                ci, cj, g = T.decode(u)
                rec, p = T.column(ci, cj) * Hg + g, T.p(ci, cj, g)
                assert 0 <= rec < records and rec not in owner
                owner[rec] = b
                places.add(p)
                assert p + ci * rrow + rbase == rec
                # neighbours in the padded arrays, z ones a group to either side
                for q in (p, p + T.pitch * Hg, p - T.pitch * Hg, p + Hg, p - Hg, p + 1, p - 1):
                    assert 0 <= q < P["pad"] <= 65535
                if T.shared(ci, cj):
                    published.add(rec)
            halos = T.halos()
            assert len(halos) <= P["halo"]
            for rec, p in halos:
                assert 0 <= rec < records and 0 < p < P["pad"] and p not in places
                wanted.add((b, rec))
            assert len({p for _, p in halos}) == len(halos)
        assert len(owner) == records
        for b, rec in wanted:
            assert rec in published and owner[rec] != b
        # every neighbour of another tile is one of the records that tile reads
        for rec, b in owner.items():
            i, j = divmod(rec // Hg, ny)
            for di, dj in ((1, 0), (-1, 0), (0, 1), (0, -1)):
                if 0 <= i + di < nx and 0 <= j + dj < ny:
                    n = ((i + di) * ny + j + dj) * Hg + rec % Hg
                    if owner[n] != b:
                        assert (b, n) in wanted
    assert planned >= (5 if maxb == 1 else 10)


def exact_smem(P, nst=13):
    return 2 * P["pad"] * 16 + P["groups"] * (32 * nst + 8) + ((P["halo"] * 6 + 15) & ~15)


SMEM = {"fp32": dc_smem, "fp64": exact_smem}
NTHREADS = {"fp32": lambda P: 512 if P["groups"] <= 512 else 384, "fp64": lambda P: 512}
