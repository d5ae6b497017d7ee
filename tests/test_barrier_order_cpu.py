"""Every order in which the two sides of the tensor-core attention (csrc/dense_attention_tc.cu) can reach their barriers, on a model:
the thread that issues copies and products, and the rows that turn scores into weights.  A wait on an mbarrier names a phase by
its parity alone, so it is right only while nobody is two phases behind."""

import pytest


def passes(over, phase):
    """What the hardware answers to a wait for ``phase`` of a barrier of which ``over`` phases are over."""
    return (over - 1) % 2 == phase % 2


def issuer(tiles, score_tiles):
    """The issuing thread of dense_attention_tc_kernel, ALONE where there are two tiles of scores."""
    yield "wait", "q", 0
    yield "wait", "k", 0
    yield "scores", 0, None
    for tile in range(tiles):
        yield "wait", ("s", tile % score_tiles), tile // score_tiles
        more = tile + 1 < tiles
        if more:
            yield "copy", "k", None
            if score_tiles == 2:
                yield "wait", "k", tile + 1
                yield "scores", tile + 1, None
        yield "wait", "v", tile
        yield "wait", "weights", tile
        yield "sums", tile, None
        yield "wait", "sums", tile
        if more:
            yield "copy", "v", None
            if score_tiles == 1:
                yield "wait", "k", tile + 1
                yield "scores", tile + 1, None


def rows(tiles, score_tiles, waits):
    for tile in range(tiles):
        yield "wait", ("s", tile % score_tiles), tile // score_tiles
        if waits and score_tiles == 2 and tile > 0:
            yield "wait", "sums", tile - 1
        yield "arrive", "weights", None
    yield "wait", "sums", tiles - 1


def giving_up(tiles, score_tiles, steps):
    """The issuer whose wait after ``steps`` of its steps has run out: it waits once more for the last of each kind that it issued."""
    done = list(issuer(tiles, score_tiles))[:steps]
    count = lambda kind, which=None: sum(step[0] == kind and which in (None, step[1]) for step in done)
    yield from done
    yield "wait", "q", 0
    yield "wait", "k", count("copy", "k")
    yield "wait", "v", count("copy", "v")
    if count("scores"):
        yield "wait", ("s", (count("scores") - 1) % score_tiles), (count("scores") - 1) // score_tiles
    if count("sums"):
        yield "wait", "sums", count("sums") - 1


def orders(programs, score_tiles):
    """What can go wrong, over all orders: waits that pass too early ("early"), sides that wait for good ("stuck"), and an issuer that
    ends before what it issued ("left").  A copy or product is asynchronous: it is under way until some later point; products
    end in the order of their issue."""
    programs = [list(program) for program in programs]
    wrong, seen = set(), set()
    start = ((0, 0), (("k", 0), ("q", 0), ("s", 0), ("s1", 0), ("sums", 0), ("v", 0), ("weights", 0)), frozenset("qkv"), ())
    name = lambda which: which if isinstance(which, str) else ("s", "s1")[which[1]]
    pending = [start]
    while pending:
        state = pending.pop()
        if state in seen:
            continue
        seen.add(state)
        places, counts, copies, products = state
        phases = dict(counts)
        moved = lambda which: tuple(sorted({**phases, which: phases[which] + 1}.items()))
        following = [(places, moved(copy), copies - {copy}, products) for copy in copies]
        if products:
            following.append((places, moved(products[0]), copies, products[1:]))
        for side, program in enumerate(programs):
            if places[side] == len(program):
                continue
            kind, which, phase = program[places[side]]
            after = tuple(place + (index == side) for index, place in enumerate(places))
            if kind == "wait":
                if passes(phases[name(which)], phase):
                    if phases[name(which)] <= phase:
                        wrong.add("early")
                        continue
                    following.append((after, counts, copies, products))
            elif kind == "copy":
                following.append((after, counts, copies | {which}, products))
            elif kind == "scores":
                following.append((after, counts, copies, products + (name(("s", which % score_tiles)),)))
            elif kind == "sums":
                following.append((after, counts, copies, products + ("sums",)))
            else:
                following.append((after, moved(which), copies, products))
        if places[0] == len(programs[0]) and (copies or products):
            wrong.add("left")
        if not following and any(place < len(program) for place, program in zip(places, programs)):
            wrong.add("stuck")
        pending.extend(following)
    return wrong


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("score_tiles", [1, 2])
def test_no_wait_ends_early_and_none_lasts(tiles, score_tiles):
    assert orders((issuer(tiles, score_tiles), rows(tiles, score_tiles, True)), score_tiles) == set()


@pytest.mark.parametrize("tiles", [2, 3, 4])
def test_the_model_sees_rows_that_do_not_wait(tiles):
    """Without the rows' wait for P V of the tile before (a late V is enough) the last wait ends early and the issuer gets stuck."""
    assert orders((issuer(tiles, 2), rows(tiles, 2, False)), 2) == {"early", "stuck"}


@pytest.mark.parametrize("tiles", [1, 2, 3, 4])
@pytest.mark.parametrize("score_tiles", [1, 2])
def test_nothing_is_under_way_when_the_issuer_has_given_up(tiles, score_tiles):
    program = list(issuer(tiles, score_tiles))
    for steps, step in enumerate(program):
        if step[0] == "wait":  # rows may go on or give up as well: only the issuer's end counts
            assert orders((giving_up(tiles, score_tiles, steps), rows(tiles, score_tiles, True)), score_tiles) <= {"stuck"}
