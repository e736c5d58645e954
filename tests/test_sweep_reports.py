"""The staged FP32 sweep's overlapping phases (csrc/tse_dc.cu dc_sweep_tma_kernel) as a
simulation of its roles: producers behind their gates and rings, consumer groups that own
stages and arrive once a warp and chunk, a reporter and a gatekeeper a block."""
import random

import pytest

HEAD, GROUP_WARPS = 16, 4


def _head(SX, H, Nc, C, nb):
    nch = -(-Nc // C)
    rounds = -(-nch // nb)
    far = -(-(SX + H + C + 16) // (nb * C))
    far += far & 1
    h = (rounds - far) // 2
    h = (HEAD if h > HEAD else 2 if h < 2 else h) & ~1
    return nch, h, h + far


class Block:
    """One block's state; a wait by parity passes as mbarrier.try_wait.parity does."""

    def __init__(self, sim, b):
        self.sim, self.b = sim, b
        S = sim
        self.mine = (S.nch - 1 - b) // S.nb + 1
        self.arrivals = [GROUP_WARPS * min(self.mine, S.first), GROUP_WARPS * (self.mine - S.first)]
        self.seg = [0, 0]                  # arrivals on seg_bar, ever
        self.gate = [0, 0]                 # completed phases of the gates
        self.reports = [(p, s) for p in range(S.phases) for s in range(S.nseg) if self.mine > (S.first if s else 0)]
        self.reported = self.opened = 0
        self.uses = [[(p, i) for p in range(S.phases) for i in range(pipe, self.mine, S.pipes)]
                     for pipe in range(S.pipes)]
        self.issued = [0] * S.pipes
        self.passed = [set() for _ in range(S.pipes)]          # gates a pipeline's producer has been through
        self.landed = [[0] * S.ring for _ in range(S.pipes)]   # completed phases of the full barriers
        self.freed = [[0] * S.ring for _ in range(S.pipes)]    # arrivals on the empty barriers
        self.flying = []
        # a group's warps: the uses of the stages it owns, in order
        self.todo = {(pipe, g, w): [u for u in range(len(self.uses[pipe])) if (u % S.ring) % S.gpp == g]
                     for pipe in range(S.pipes) for g in range(S.gpp) for w in range(GROUP_WARPS)}
        self.at = dict.fromkeys(self.todo, 0)
        self.err = False

    def parity(self, completed, phase):
        if (completed & 1) == (phase & 1):
            return False
        assert completed == phase + 1, "a parity wait passed early or was lapped"
        return True

    def produce(self, pipe):
        S = self.sim
        if self.issued[pipe] == len(self.uses[pipe]):
            return False
        p, i = self.uses[pipe][self.issued[pipe]]
        need = []
        if i == pipe:
            need.append(0)
        if S.nseg > 1 and i >= S.head and i - S.pipes < S.head:
            need.append(1)
        for s in need:
            if (p, s) not in self.passed[pipe]:
                if not self.parity(self.gate[s], p):
                    return False
                self.passed[pipe].add((p, s))
        u = self.issued[pipe]
        s = u % S.ring
        if u >= S.ring and not self.parity(self.freed[pipe][s] // GROUP_WARPS, u // S.ring - 1):
            return False
        q = self.b + i * S.nb
        if p:   # the windows are read now
            for r in range(max(0, q - S.reach), min(S.nch, q + S.reach + 1)):
                assert S.swept[p - 1][r] == GROUP_WARPS, "a window copied before it was written"
        self.issued[pipe] += 1
        self.flying.append((pipe, s))
        return True

    def land(self, rng):
        if not self.flying:
            return False
        pipe, s = self.flying.pop(rng.randrange(len(self.flying)))
        self.landed[pipe][s] += 1
        return True

    def consume(self, k):
        S = self.sim
        if self.at[k] == len(self.todo[k]):
            return False
        pipe = k[0]
        u = self.todo[k][self.at[k]]
        s = u % S.ring
        if not self.parity(self.landed[pipe][s], u // S.ring):
            return False
        p, i = self.uses[pipe][u]
        S.swept[p][self.b + i * S.nb] += 1
        self.freed[pipe][s] += 1
        t = 1 if i >= S.first else 0
        self.seg[t] += 1
        assert self.seg[t] <= (p + 1) * self.arrivals[t], "arrivals of a phase before the one before is done"
        self.at[k] += 1
        return True

    def report(self):
        if self.reported == len(self.reports):
            return False
        p, s = self.reports[self.reported]
        if not self.parity(self.seg[s] // self.arrivals[s], p):
            return False
        self.sim.count[s] += 1
        self.reported += 1
        return True

    def open(self):
        S = self.sim
        if self.opened == S.phases * S.nseg:
            return False
        p, s = divmod(self.opened, S.nseg)
        if S.count[s] < p * S.blocks[s]:
            return False
        self.gate[s] += 1
        self.opened += 1
        return True

    def done(self):
        return (all(self.at[k] == len(self.todo[k]) for k in self.todo) and self.reported == len(self.reports)
                and self.opened == self.sim.phases * self.sim.nseg)


class Sim:
    def __init__(self, shape, nb, C, ring, pipes, groups, phases):
        nx, ny, nz = shape
        H = (nz + 1) // 2
        SX, Nc = ny * H, nx * ny * H
        self.nb = max(1, min(nb, -(-Nc // C)))
        self.nch, self.head, self.first = _head(SX, H, Nc, C, self.nb)
        self.nseg = 2 if self.nch > self.first * self.nb else 1
        self.ring, self.pipes, self.gpp, self.phases = ring, pipes, groups // pipes, phases
        self.blocks = [min(self.nb, self.nch - s * self.first * self.nb) for s in range(self.nseg)]
        self.count = [0, 0]
        self.reach = -(-(max(SX, H + 1) + 8) // C)
        self.swept = [[0] * self.nch for _ in range(phases)]
        self.block = [Block(self, b) for b in range(self.nb)]

    def run(self, rng, bad=None, when=0):
        """Until nothing moves; block ``bad`` gives up after ``when`` of its steps."""
        moves = 0
        live = [b for b in self.block]
        while live:
            moved = False
            rng.shuffle(live)
            for B in live:
                if B.b == bad and moves >= when:
                    B.err = True
                if B.err:
                    continue
                acts = [B.report, B.open, lambda: B.land(rng)] + [lambda pipe=pipe: B.produce(pipe) for pipe in
                                                                  range(self.pipes)]
                acts += [lambda k=k: B.consume(k) for k in B.todo]
                rng.shuffle(acts)
                for act in acts[:rng.randint(1, len(acts))]:
                    did = act()
                    moved = moved or did
                    moves += did and B.b == bad
            live = [B for B in live if not B.done() and not B.err]
            if not moved and all(B.err or not any((B.report(), B.open(), B.land(rng))) and
                                 not any([B.produce(x) for x in range(self.pipes)]) and
                                 not any([B.consume(k) for k in B.todo]) for B in live):
                break
        return [not B.err and B.done() for B in self.block]


FORMS = [(2, 2), (2, 4), (1, 2)]   # pipelines, consumer groups: 8 warps, 16 warps, one pipeline
CASES = [((40, 36, 50), 5), ((9, 1, 31), 2), ((30, 30, 11), 7), ((20, 40, 64), 3), ((60, 30, 40), 2)]


@pytest.mark.parametrize("pipes,groups", FORMS)
def test_reports_and_gates_order_the_phases(pipes, groups):
    rng = random.Random(10 * pipes + groups)
    for shape, nb in CASES:
        sim = Sim(shape, nb, 256, rng.choice((2, 3, 4)), pipes, groups, 5)
        assert all(sim.run(rng)), "no progress"
        assert all(x == GROUP_WARPS for phase in sim.swept for x in phase)
        assert [sim.count[s] for s in range(sim.nseg)] == [5 * x for x in sim.blocks]


@pytest.mark.parametrize("pipes,groups", FORMS)
def test_a_block_that_gave_up_is_known_at_the_end(pipes, groups):
    """The leader (block 0) may finish all its phases though another block gave
    up in the last ones: its own flag does not tell, the blocks' marks as they
    leave do."""
    rng = random.Random(pipes + groups)
    own_flag_passes = 0
    for n in range(60):
        shape, nb = CASES[n % len(CASES)]
        sim = Sim(shape, nb, 256, 3, pipes, groups, 2)
        if sim.nb < 2:
            continue
        bad = rng.randrange(1, sim.nb)
        steps = sum(len(x) for x in sim.block[bad].todo.values())
        ended = sim.run(rng, bad, rng.randint(1, 2 * steps))
        if sim.block[bad].err:
            assert not ended[bad] and not all(ended)
            own_flag_passes += ended[0]
    assert own_flag_passes > 0
