"""Model of one block of a run of matmul_q steps (lex_gpu_b200/csrc/matmul_q_chain_sm100.cuh) under random interleavings.

The copy engine (codes, the scale bytes a group of four stages at a time and a group ahead of the codes, digit rows from the launch
ahead), two sets of scale warps that take the even and the odd stages, the MMA warp and the epilogue, with parity waits on barriers
that count as the kernel's do.  A scale warp that meets a negative scale byte waits for the stage's codes; one that meets a NaN byte
leaves a flag for the epilogue of its part of K.  The model checks that no parity wait passes before the phase it stands for, that
everything ends, and that every flag is found by the part it belongs to and by no other.
"""
import random

import pytest

GROUP, WS_SLOTS = 4, 3


class Bar:
    def __init__(self, count=1):
        self.count = self.pending = count
        self.done = 0

    def arrive(self):
        self.pending -= 1
        assert self.pending >= 0
        if not self.pending:
            self.pending, self.done = self.count, self.done + 1

    def passes(self, parity):
        return (self.done & 1) != parity


def run(tiles, S, seed, negative=(), nan=(), flags="parts", held_back=False):
    """`tiles`: (stages, stages per part of K); `negative`, `nan`: the stages with such a scale byte.  flags="sets": one flag per set
    of accumulators behind a parity wait for the part two before.  `held_back`: the copy engine asks for a stage's scale bytes ahead of
    its codes and digit rows.  -> parts found flagged, most parts open at once, errors."""
    rnd = random.Random(seed)
    stages, parts, groups = [], 0, 0                          # (part, first of a group, group, a tile's stage), ...
    group_stages = []
    for kb_all, per in tiles:
        for kb in range(kb_all):
            stages.append((parts + kb // per, kb % per == per - 1 or kb + 1 == kb_all, groups + kb // GROUP))
        for g0 in range(0, kb_all, GROUP):
            group_stages.append([len(stages) - kb_all + kb for kb in range(g0, min(kb_all, g0 + GROUP))])
        parts += (kb_all + per - 1) // per
        groups += (kb_all + GROUP - 1) // GROUP
    raw_full, empty, prep_full = ([Bar(c) for _ in range(S)] for c in (2, 1, 1))      # raw_full: codes, digit rows
    ws_full, ws_empty = ([Bar(c) for _ in range(WS_SLOTS)] for c in (1, 2))
    acc_full, acc_empty = [Bar(), Bar()], [Bar(), Bar()]
    errors, found, word, stored, most = [], [], [0], [-1], [0]

    def wait(bar, phase, what):                               # for the barrier's `phase`-th completion (-1: none needed)
        while not bar.passes(phase & 1):
            yield
        if bar.done < phase + 1:
            errors.append("passed early: " + what)

    def copy():
        issued = begun = digits = 0
        ordered = False                                       # the launch ahead has been waited for
        for i, (_, _, g) in enumerate(stages):
            yield from wait(empty[i % S], i // S - 1, f"copy empty {i}")
            starts = i == group_stages[g][0]
            begun += starts
            for what in ("groups", "stage") if held_back else ("stage", "groups"):
                if what == "stage":
                    raw_full[i % S].arrive()
                    yield
                    ordered |= i + 1 >= S or i + 1 == len(stages) or (starts and begun >= WS_SLOTS and not held_back)
                    for d in range(digits, i + 1 if ordered else digits):
                        raw_full[d % S].arrive()
                        digits = d + 1
                    continue
                while starts and issued < min(begun + 1, groups):
                    ordered |= issued >= WS_SLOTS
                    yield from wait(ws_empty[issued % WS_SLOTS], issued // WS_SLOTS - 1, f"copy ws_empty {issued}")
                    ws_full[issued % WS_SLOTS].arrive()
                    issued += 1

    def scale(par):
        for i, (p, _, g) in enumerate(stages):
            if i % 2 != par:
                continue
            yield from wait(empty[i % S], i // S - 1, f"scale empty {i}")
            yield from wait(ws_full[g % WS_SLOTS], g // WS_SLOTS, f"scale ws_full {g}")
            most[0] = max(most[0], p - stored[0])
            if i + 2 not in group_stages[g]:                  # this set's last stage of the group
                ws_empty[g % WS_SLOTS].arrive()
            yield
            if i in negative:
                yield from wait(raw_full[i % S], i // S, f"scale raw_full {i}")
            if i in nan:
                if flags == "parts":
                    word[0] |= 1 << (p & 31)
                else:
                    while p >= 2 and not acc_empty[p & 1].passes(((p >> 1) - 1) & 1):
                        yield
                    word[0] |= 1 << (p & 1)
            yield
            prep_full[i % S].arrive()

    def mma():
        first = True
        for i, (p, ends, _) in enumerate(stages):
            if first:
                yield from wait(acc_empty[p & 1], (p >> 1) - 1, f"mma acc_empty {p}")
            yield from wait(raw_full[i % S], i // S, f"mma raw_full {i}")
            yield from wait(prep_full[i % S], i // S, f"mma prep_full {i}")
            yield
            empty[i % S].arrive()
            if ends:
                acc_full[p & 1].arrive()
            first = ends

    def epilogue():
        for p in range(parts):
            yield from wait(acc_full[p & 1], p >> 1, f"epilogue {p}")
            for _ in range(rnd.randint(0, 12)):
                yield
            bit = 1 << (p & (31 if flags == "parts" else 1))
            if word[0] & bit:
                found.append(p)
                word[0] &= ~bit
            yield
            stored[0] = p
            acc_empty[p & 1].arrive()

    actors = [copy(), scale(0), scale(1), mma(), epilogue()]
    weight = [rnd.random() + 0.05 for _ in actors]
    live = list(range(len(actors)))
    for _ in range(400 * len(stages) + 20_000):
        if not live or errors:
            break
        i = rnd.choices(live, [weight[a] for a in live])[0]
        try:
            next(actors[i])
        except StopIteration:
            live.remove(i)
    if live and not errors:
        errors.append("nothing moves")
    return found, most[0], {stages[i][0] for i in nan}, errors


SHAPES = [[(2, 2)] * 12, [(3, 3)] * 10, [(4, 4)] * 8, [(6, 6)] * 5, [(7, 7)] * 4, [(22, 5)] * 4, [(68, 9)] + [(2, 2)] * 6,
          [(20, 4), (7, 7), (6, 6), (3, 3), (3, 3), (2, 2), (2, 2), (2, 2)], [(3, 1)] * 10]


@pytest.mark.parametrize("S", [7, 8])
@pytest.mark.parametrize("tiles", SHAPES)
def test_a_flag_is_found_by_its_own_part(tiles, S):
    for seed in range(15):
        rnd = random.Random(1000 + seed)
        total = sum(kb for kb, _ in tiles)
        nan = set(rnd.sample(range(total), rnd.randint(1, 4)))
        found, most, want, errors = run(tiles, S, seed, nan=nan)
        assert not errors and set(found) == want and len(found) == len(want)
        assert most <= S + 2                                  # parts open at once: the flags are bits of one 32-bit word


def test_flags_per_accumulator_set_would_be_found_by_another_part():
    wrong = 0
    for seed in range(20):
        found, _, want, _ = run([(2, 2)] * 12, 8, seed, nan={8}, flags="sets")      # the block's fifth tile of two stages
        wrong += set(found) != want
    assert wrong


@pytest.mark.parametrize("S", [7, 8])
@pytest.mark.parametrize("tiles", SHAPES)
def test_negative_scale_bytes_wait_for_nothing_that_is_held_back(tiles, S):
    for seed in range(15):
        rnd = random.Random(2000 + seed)
        total = sum(kb for kb, _ in tiles)
        negative = {0, 1} | set(rnd.sample(range(total), total // 3))
        nan = set(rnd.sample(range(total), 2))
        found, _, want, errors = run(tiles, S, seed, negative=negative, nan=nan)
        assert not errors and set(found) == want


@pytest.mark.parametrize("tiles", [[(3, 3)] * 10, [(6, 6)] * 5, [(7, 7)] * 4])
def test_digit_rows_held_back_would_stop_a_run_of_few_stages(tiles):
    assert run(tiles, 8, 0, negative={0}, held_back=True)[3] == ["nothing moves"]
