"""The staged sweep's overlapping phases (csrc/tse_dc.cuh sweep_head, dc_sweep_tma_kernel)
on the CPU: a restatement of which rounds a phase may begin with, what a chunk's windows
reach, and of the reports and gates that replace a device-wide barrier."""
import random

import pytest

HEAD, GROUP_WARPS, WARPS = 16, 4, 8


def _layout(nx, ny, nz):
    H = (nz + (nz & 1)) // 2
    return H, ny * H, nx * ny * H


def _head(H, SX, Nc, C, nb):
    nch = -(-Nc // C)
    rounds = -(-nch // nb)
    far = -(-(SX + H + C + 16) // (nb * C))
    far += far & 1
    h = (rounds - far) // 2
    h = HEAD if h > HEAD else 2 if h < 2 else h
    h &= ~1
    return nch, rounds, far, h, h + far


def _cases():
    rng = random.Random(9)
    out = [(256, 256, 128, 148), (100, 100, 100, 148), (512, 512, 256, 148), (64, 64, 64, 148),
           (3, 2, 1000, 5), (1, 2, 3000, 3), (9, 1, 31, 1), (40, 36, 50, 148)]
    return out + [(rng.randint(1, 90), rng.randint(1, 90), rng.randint(1, 200), rng.choice((1, 5, 37, 148)))
                  for _ in range(40)]


@pytest.mark.parametrize("C", [256, 512, 1024])
def test_the_head_reads_and_writes_only_what_the_first_report_covers(C):
    for nx, ny, nz, cap in _cases():
        H, SX, Nc = _layout(nx, ny, nz)
        nb = max(1, min(cap, -(-Nc // C)))
        nch, rounds, far, head, first = _head(H, SX, Nc, C, nb)
        assert head >= 2 and head % 2 == 0 and first % 2 == 0
        for q in range(nch):
            hi = min(Nc - 1, q * C + C + max(SX, H) + 7)
            if q // nb < head:
                assert (hi // C) // nb < first
        for s in range(2 if nch > first * nb else 1):
            have = {q % nb for q in range(nch) if (q // nb >= first) == bool(s)} if s or nch > first * nb \
                else {q % nb for q in range(nch)}
            assert len(have) == min(nb, nch - s * first * nb)


def test_phases_follow_each_other_without_a_barrier():
    """Random progress of the consumer warps, reporters and gatekeepers of a
    few blocks through several phases: nothing deadlocks, a report is counted
    once a block and phase and only when all of that block's warps with chunks
    there have arrived, and a chunk is swept only after every chunk of the
    other colour that its windows reach."""
    rng = random.Random(2)
    for nx, ny, nz, cap in [(40, 36, 50, 5), (9, 1, 31, 2), (30, 30, 11, 7), (20, 40, 64, 3), (60, 30, 40, 2)]:
        H, SX, Nc = _layout(nx, ny, nz)
        C = 256
        nb = max(1, min(cap, -(-Nc // C)))
        nch, rounds, far, head, first = _head(H, SX, Nc, C, nb)
        nseg = 2 if nch > first * nb else 1
        phases = 4
        mine = [(nch - 1 - b) // nb + 1 for b in range(nb)]
        blocks = [min(nb, nch - s * first * nb) for s in range(nseg)]
        warps = lambda b, s: WARPS if (mine[b] - first if s else min(mine[b], first)) >= 2 else GROUP_WARPS
        reach = -(-(max(SX, H + 1) + C + 8) // C)
        swept = [[0] * nch for _ in range(phases)]        # warps done with a chunk
        arrived = [[0] * nseg for _ in range(nb)]         # arrivals on seg_bar, ever
        count = [0] * nseg
        reported = [0] * nb      # (phase, s) pairs the reporter has made, in order
        gates = [0] * nb         # (phase, s) pairs the gatekeeper has opened
        work = {(b, g, w): [(p, i) for p in range(phases) for i in range(g, mine[b], 2)]
                for b in range(nb) for g in range(2) for w in range(GROUP_WARPS)}
        at = dict.fromkeys(work, 0)
        last = dict.fromkeys(work)   # (phase, report) of the warp's last chunk
        rep = [[(p, s) for p in range(phases) for s in range(nseg) if mine[b] > (first if s else 0)]
               for b in range(nb)]
        idle = 0
        while any(at[k] < len(work[k]) for k in work):
            idle += 1
            assert idle < 200000, "no progress"
            b = rng.randrange(nb)
            kind = rng.randrange(3)
            if kind == 0 and gates[b] < phases * nseg:
                p, s = divmod(gates[b], nseg)
                if count[s] >= p * blocks[s]:
                    gates[b] += 1
            elif kind == 1 and reported[b] < len(rep[b]):
                p, s = rep[b][reported[b]]
                assert arrived[b][s] <= (p + 1) * warps(b, s)
                if arrived[b][s] == (p + 1) * warps(b, s):
                    reported[b] += 1
                    count[s] += 1
            elif kind == 2:
                k = (b, rng.randrange(2), rng.randrange(GROUP_WARPS))
                if at[k] == len(work[k]):
                    continue
                p, i = work[k][at[k]]
                need = p * nseg + (2 if nseg > 1 and i >= head else 1)
                if gates[b] < need:
                    continue
                q = b + i * nb
                if p:
                    for r in range(max(0, q - reach), min(nch, q + reach + 1)):
                        assert swept[p - 1][r] == GROUP_WARPS
                swept[p][q] += 1
                at[k] += 1
                s = 1 if nseg > 1 and i >= first else 0
                nxt = work[k][at[k]] if at[k] < len(work[k]) else None
                if nxt is None or nxt[0] != p or (nseg > 1 and (nxt[1] >= first) != bool(s)):
                    arrived[b][s] += 1
                idle = 0
        assert all(count[s] <= phases * blocks[s] for s in range(nseg))


def test_record_blocks_are_aligned_and_inside_their_array():
    """A chunk's record block (records, r', flags) is one copy: 16-byte
    aligned, a multiple of 16 bytes, inside the colour's array for every
    compiled chunk size, and every cell's parts lie where the copy puts them."""
    rng = random.Random(3)
    for Nc in [1, 2, 255, 256, 257, 511, 512, 1023, 1024, 1025] + [rng.randint(1, 200000) for _ in range(40)]:
        floats = ((Nc + 1023) >> 10) * (29 << 8)
        assert 2 * floats * 4 % 16 == 0            # the second colour and the corrections after it
        for ks in (8, 9, 10):
            C, block = 1 << ks, 29 << (ks - 2)
            assert block * 4 % 16 == 0 and block * 4 == 29 * C
            for q in range(-(-Nc // C)):
                assert (q + 1) * block <= floats
            for m in (0, Nc // 2, Nc - 1):
                o = m & (C - 1)
                base = (m >> ks) * block
                rec, rp, flag = base + 6 * o, base + 6 * C + o, 4 * (base + 7 * C) + o
                assert rec * 4 % 8 == 0 and rec + 6 <= base + 6 * C
                assert rp < base + 7 * C and flag < 4 * (base + block)


@pytest.mark.parametrize("ring,groups", [(2, 1), (3, 1), (4, 1), (2, 2), (3, 2), (4, 2)])
def test_parity_waits_never_pass_early(ring, groups):
    """The stages of one pipeline: an in-order producer, copies that land in
    any order, consumer groups that test a stage's full barrier by parity only.
    A stage belongs to one group, so no group ever reads a use whose copies
    have not landed and no barrier gets an arrival too many -- also over
    phases whose chunk count is odd.  (With chunks dealt to the groups in turn
    it happens within a few hundred tries; the second loop shows it.)"""
    def run(by_stage, rng, phases=6, pmine=5):
        total = phases * pmine
        full = [0] * ring        # completed phases of each full barrier
        empty = [0] * ring
        issued, landing = 0, []
        if by_stage:
            mine = [[u for u in range(total) if (u % ring) % groups == g] for g in range(groups)]
        else:
            mine = [[u for u in range(total) if (u % pmine) % groups == g] for g in range(groups)]
        at = [0] * groups
        for _ in range(20000):
            if all(at[g] == len(mine[g]) for g in range(groups)):
                return True
            what = rng.randrange(3)
            if what == 0 and issued < total:
                s = issued % ring
                # mbarrier.try_wait.parity: true once the current phase's parity differs
                if issued < ring or (empty[s] & 1) != ((issued // ring - 1) & 1):
                    if issued >= ring and empty[s] != issued // ring:
                        return False
                    landing.append(issued)
                    issued += 1
            elif what == 1 and landing:
                u = landing.pop(rng.randrange(len(landing)))
                full[u % ring] += 1
            elif what == 2:
                g = rng.randrange(groups)
                if at[g] < len(mine[g]):
                    u = mine[g][at[g]]
                    s = u % ring
                    if (full[s] & 1) != ((u // ring) & 1):
                        if full[s] != u // ring + 1:
                            return False            # read before its copies landed
                        empty[s] += 1
                        at[g] += 1
        return False

    rng = random.Random(ring * 10 + groups)
    assert all(run(True, rng) for _ in range(300))
    if groups == 2 and ring == 4:
        assert not all(run(False, rng) for _ in range(300))
