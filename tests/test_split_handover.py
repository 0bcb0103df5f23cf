"""Hand-overs of the split tensor form (mc_tcws_kernel with SPLIT), on the CPU.

A wait on an mbarrier names a phase by its parity alone: it passes when the
current phase's parity differs, so a role that falls a phase behind (or runs a
phase ahead) takes another phase for its own.  The roles of one CTA (generator
with its publisher, copy warp, two MMA issuers, epilogue) are run here as
coroutines under schedules that hold one of them up; each wait knows which
phase it means, and one that passes on another phase, a read of a tile slot
that was published again, or a wait that never passes is an error.  The barrier
counts and the issuers' steps are read from the kernel's source.
"""
import os
import random
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-montecarlo-risk_gb300", "csrc",
                   "rg_mc_tc.cu")
ISSUERS, TILE_SLOTS = 2, 3


class Wrong(Exception):
    pass


class Bar:
    def __init__(self, count):
        self.count, self.left, self.done = count, count, 0  # done: completed phases

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left, self.done = self.count, self.done + 1

    def passes(self, phase):
        """A parity wait for the end of `phase` (-1: the fresh barrier's)."""
        return (self.done & 1) != (phase & 1)

    def check(self, phase, what):
        if self.done != phase + 1:
            raise Wrong(f"{what}: wait for phase {phase} passed after {self.done} phases")


def kts(mt, n_mt, n_kt):
    return n_kt if mt == n_mt - 1 else min(n_kt, 2 * (mt + 1))


def simulate(rule, n_mt, n_kt, z_slots, stages, tiles, seed):
    rng = random.Random(seed)
    # the Lhat stages in rings: one an issuer, or one for both
    if rule["own_rings"]:
        rings = [range((stages + 1) // 2), range((stages + 1) // 2, stages)]
    else:
        rings = [range(stages)] * 2
    empty = [Bar(1) for _ in range(stages)]
    full = [Bar(1) for _ in range(stages)]
    zfull = [Bar(1) for _ in range(z_slots)]
    zempty = [Bar(ISSUERS) for _ in range(z_slots)]
    acc_full = [Bar(1) for _ in range(n_mt)]
    acc_free = [Bar(1) for _ in range(n_mt)]
    pub = [Bar(1) for _ in range(TILE_SLOTS)]
    slot_free = [Bar(rule["slot_free"]) for _ in range(TILE_SLOTS)]
    s_tile = [None] * TILE_SLOTS
    copies = []                          # copies in flight (stage, use): they land in any order
    commits = [[], []]                   # per issuer: MMAs and commits complete in order

    def generator():
        def publish(j):
            yield slot_free[j % TILE_SLOTS], j // TILE_SLOTS - 1, "slot_free"
            s_tile[j % TILE_SLOTS] = j if j < tiles else -1
            pub[j % TILE_SLOTS].arrive()
        yield from publish(0)
        for j in range(tiles):
            yield from publish(j + 1)
            yield pub[j % TILE_SLOTS], j // TILE_SLOTS, "tile_pub"
            for kt in range(n_kt):
                g = j * n_kt + kt
                yield zempty[g % z_slots], g // z_slots - 1, "zempty"
                zfull[g % z_slots].arrive()

    def tile_of(j):
        yield pub[j % TILE_SLOTS], j // TILE_SLOTS, "tile_pub"
        yield None
        if s_tile[j % TILE_SLOTS] != (j if j < tiles else -1):
            raise Wrong("tile slot published again before it was read")

    def copy_warp():
        made = [0, 0]
        for j in range(tiles):
            yield from tile_of(j)
            for kt in range(n_kt):
                for mt in range(n_mt):
                    if kt < kts(mt, n_mt, n_kt):
                        me = mt % 2 if rule["own_rings"] else 0
                        stage, use = rings[me][made[me] % len(rings[me])], made[me] // len(rings[me])
                        yield empty[stage], use - 1, "empty_bar"
                        copies.append((stage, use))
                        made[me] += 1
        yield from tile_of(tiles)

    def issuer(me):
        i, uses = 0, [0] * n_mt
        for j in range(tiles):
            yield from tile_of(j)
            for kt in range(n_kt):
                g = j * n_kt + kt
                yield zfull[g % z_slots], g // z_slots, "zfull"
                for mt in range(n_mt):
                    if kt >= kts(mt, n_mt, n_kt):
                        continue
                    stage, use = rings[me][i % len(rings[me])], i // len(rings[me])
                    if mt % 2 != me:
                        i += 0 if rule["own_rings"] else 1  # the other issuer's pair, unseen
                        continue
                    if kt == 0:
                        yield acc_free[mt], uses[mt] - 1, "acc_free"
                    yield full[stage], use, "full_bar"
                    commits[me].append(empty[stage])
                    if kt == kts(mt, n_mt, n_kt) - 1:
                        commits[me].append(acc_full[mt])
                        uses[mt] += 1
                    i += 1
                commits[me].append(zempty[g % z_slots])
            if rule["issuer_frees"]:
                slot_free[j % TILE_SLOTS].arrive()
        yield from tile_of(tiles)

    def epilogue():
        for j in range(tiles):
            yield from tile_of(j)
            for mt in range(n_mt):
                yield acc_full[mt], j, "acc_full"
                acc_free[mt].arrive()
            slot_free[j % TILE_SLOTS].arrive()
        yield from tile_of(tiles)

    roles = {"generator": generator(), "copy": copy_warp(), "issuer 0": issuer(0), "issuer 1": issuer(1),
             "epilogue": epilogue()}
    waits = {name: None for name in roles}
    held, hold = None, 0
    while roles or copies or any(commits):
        if hold == 0:
            held, hold = rng.choice(list(roles) + [None, "lands"]), rng.randint(1, 400)
        hold -= 1
        ready = [n for n in roles if waits[n] is None or waits[n][0].passes(waits[n][1])]
        landing = [("land", c) for c in copies] + [("commit", k) for k in range(2) if commits[k]]
        free = [n for n in ready if n != held] + ([] if held == "lands" else landing)
        if not free:
            if not ready and not landing:
                raise Wrong("a wait that never passes: " + str({n: waits[n][2] for n in roles}))
            hold = 0
            continue
        act = rng.choice(free)
        if isinstance(act, tuple):
            if act[0] == "land":
                copies.remove(act[1])
                full[act[1][0]].check(act[1][1] - 1, "a copy into a stage in use")
                full[act[1][0]].arrive()
            else:
                commits[act[1]].pop(0).arrive()
            continue
        if waits[act] is not None:
            waits[act][0].check(waits[act][1], f"{act}, {waits[act][2]}")
        try:
            waits[act] = next(roles[act])
        except StopIteration:
            del roles[act]


def _rule():
    """The counts and steps of the kernel as it stands."""
    with open(SRC) as f:
        text = f.read()
    kernel = text[text.index("mc_tcws_kernel(const __grid_constant__"):]

    count = re.search(r"mbar_init\(&slot_free\[s\], ([^;]*)\);", kernel).group(1)
    count = count.replace("SPLIT ? ", "").split(" : ")[0].replace("kIssuers", str(ISSUERS))
    copy = kernel[kernel.index("= Lhat producer ="):kernel.index("MMA issue (and")]
    issuer = kernel[kernel.index("MMA issue (and"):kernel.index("= epilogue (warps 0-3) =")]
    return dict(slot_free=sum(int(t) for t in count.split("+")), issuer_frees="mbar_arrive(&slot_free[" in issuer,
                own_rings="kRing0" in copy and "full_bar[ring0 + rs]" in issuer)


# row tiles, K tiles, Z slots, Lhat stages: N <= 64 and <= 127 at 128 and at 96 or 64 paths, then one of each row-tile count
SHAPES = [(1, 1, 3, 4), (1, 1, 4, 4), (1, 1, 4, 5), (1, 2, 3, 4), (1, 2, 4, 4), (2, 3, 3, 4), (3, 5, 3, 4), (4, 8, 3, 4),
          (5, 9, 4, 4), (6, 10, 4, 5)]


@pytest.mark.parametrize("n_mt,n_kt,z_slots,stages", SHAPES)
def test_no_role_takes_another_phase(n_mt, n_kt, z_slots, stages):
    rule = _rule()
    for seed in range(40):
        simulate(rule, n_mt, n_kt, z_slots, stages, 14 if n_kt < 4 else 5, seed)


@pytest.mark.parametrize("weaker,shape", [
    (dict(slot_free=1, issuer_frees=False), (1, 1, 4, 4)),  # the epilogue alone frees a tile slot
    (dict(own_rings=False), (5, 9, 4, 4)),                  # the other issuer's pairs stepped over unseen
])
def test_the_model_finds_a_missing_hand_over(weaker, shape):
    sound = dict(slot_free=1 + ISSUERS, issuer_frees=True, own_rings=True)
    with pytest.raises(Wrong):
        for seed in range(400):
            simulate(dict(sound, **weaker), *shape, 14, seed)
