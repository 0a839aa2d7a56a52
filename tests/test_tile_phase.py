"""The barriers of the attention kernels that walk tiles of keys (``csrc/tile_phase.h``), in every order of events.

A model of one block: the loader of V, the issuing thread, the tensor cores (what was issued completes in order, at any
time), and two softmax warps, each of which can be held up anywhere.  An mbarrier is what the hardware has: a count of
completed phases of which a wait sees the parity only.  Which barrier and which parity stand for a tile comes from the
kernels' own header, compiled here by the host's compiler.  The walk visits every state that any schedule can reach and
reports a wait that was passed before what it waits for had happened, or a state in which nothing can move."""

import ctypes
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qwen3_from_scratch_b200", "csrc")
WARPS = 2


@pytest.fixture(scope="module")
def header(tmp_path_factory):
    compiler = shutil.which("g++") or shutil.which("c++")
    if compiler is None:
        pytest.skip("no host compiler")
    folder = tmp_path_factory.mktemp("tile_phase")
    source, library = folder / "shim.cpp", folder / "shim.so"
    source.write_text('#include "tile_phase.h"\n'
                      'extern "C" int slot(int j) { return q3::tile_slot(j); }\n'
                      'extern "C" int parity(int j) { return (int)q3::tile_parity(j); }\n')
    subprocess.run([compiler, "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(library), str(source)], check=True)
    lib = ctypes.CDLL(str(library))
    return lib.slot, lib.parity


class Fault(Exception):
    pass


def walk(n, slot, parity, hand_on=None, behind=False, ragged=False):
    """Every state of a block of ``n`` tiles.  ``slot``, ``parity``: of a tile on ``pv_done`` and, unless ``hand_on`` gives
    another pair of functions, on ``p_ready`` (the other barriers are pairs in all forms).  ``behind``: the warps follow the products one tile behind, after they
    have handed their tile on.  ``ragged``: the last tile's V is waited for by the warps too.  Raises ``Fault``."""
    p_slot, p_parity = hand_on or (slot, parity)
    # issuing thread: S 0, then for every j: S j + 1, wait for the probabilities of j, wait for V of j, P V of j
    program = [("S", 0)]
    for j in range(n):
        program += [("S", j + 1)] if j + 1 < n else []
        program += [("p", j), ("v", j), ("PV", j)]
    # a softmax warp: scores, meeting, perhaps a rescale (which waits for the product before), V, hand on, perhaps follow
    warp = []
    for j in range(n):
        warp += [("s", j), ("meet", j)] + ([("rescale", j - 1)] if j else []) + ([("v", j)] if ragged and j == n - 1 else [])
        warp += [("arrive", j)] + ([("wait", j - 1)] if behind and j else [])
    warp += [("wait", n - 1)]

    def passes(done, p):  # a wait for parity p, where `done` phases are over
        return (done + 1) & 1 == p

    # state: issuing thread's place, operations completed by the tensor cores (of those issued), V tiles asked for, V tiles
    # landed (two can be on their way, in either order: a set), arrivals on p_ready in sum, the warps' places
    start = (0, 0, 0, frozenset(), 0, (0,) * WARPS)
    seen, todo = {start}, [start]
    tensor_ops = [op for op in program if op[0] in ("S", "PV")]
    place_of = {op: i for i, op in enumerate(tensor_ops)}
    while todo:
        state = todo.pop()
        at, completed, asked, landed, arrived, warps = state
        issued = sum(op[0] in ("S", "PV") for op in program[:at])
        over = lambda op: place_of[op] < completed  # noqa: E731

        def phases(kind, of_slot, slot_of):
            return sum(over((kind, j)) for j in range(n) if slot_of(j) == of_slot)

        def pv_wait(j, passed_on):
            """Whether the wait for the product of tile j can be passed now; a fault if it must not."""
            if not passes(phases("PV", slot(j), slot), parity(j)):
                return False
            if not over(("PV", j)):
                raise Fault(f"{passed_on}: the wait for P V of tile {j} of {n} was passed before it was over")
            return True

        def v_wait(j):
            if not passes(sum(slot2(i) == slot2(j) for i in landed), parity2(j)):
                return False
            if j not in landed:
                raise Fault(f"the wait for V of tile {j} was passed before it had landed")
            return True

        slot2, parity2 = (lambda j: j & 1), (lambda j: j >> 1 & 1)
        moves = []
        if completed < issued:
            moves.append((at, completed + 1, asked, landed, arrived, warps))
        if asked < n and (asked < 2 or over(("PV", asked - 2))):
            moves.append((at, completed, asked + 1, landed, arrived, warps))
        for j in range(asked):
            if j not in landed:
                moves.append((at, completed, asked, landed | {j}, arrived, warps))
        if at < len(program):
            kind, j = program[at]
            go = True
            if kind == "p":
                # arrivals come in whole rounds of WARPS: round j is tile j's, on the barrier of its slot
                rounds = arrived // WARPS
                go = passes(sum(p_slot(i) == p_slot(j) for i in range(rounds)), p_parity(j))
                if go and rounds <= j:
                    raise Fault(f"the issuing thread passed the wait for the probabilities of tile {j} too early")
            elif kind == "v":
                go = v_wait(j)
            elif kind == "S" and j >= 2 and not over(("PV", j - 2)) and ("PV", j - 2) not in tensor_ops[:issued]:
                raise Fault(f"scores of tile {j} issued ahead of the product that reads their place")
            if go:
                moves.append((at + 1, completed, asked, landed, arrived, warps))
        for w in range(WARPS):
            if warps[w] == len(warp):
                continue
            kind, j = warp[warps[w]]
            step = warps[:w] + (warps[w] + 1,) + warps[w + 1:]
            if kind == "s":
                if passes(phases("S", slot2(j), slot2), parity2(j)):
                    if not over(("S", j)):
                        raise Fault(f"the wait for the scores of tile {j} was passed before they were ready")
                    moves.append((at, completed, asked, landed, arrived, step))
            elif kind == "meet":  # the named barrier: all warps leave it together
                if all(p == warps[w] for p in warps):
                    moves.append((at, completed, asked, landed, arrived, tuple(p + 1 for p in warps)))
            elif kind == "rescale":  # or not
                moves.append((at, completed, asked, landed, arrived, step))
                if pv_wait(j, "rescale"):
                    moves.append((at, completed, asked, landed, arrived, step))
            elif kind == "v":
                if v_wait(j):
                    moves.append((at, completed, asked, landed, arrived, step))
            elif kind == "arrive":
                moves.append((at, completed, asked, landed, arrived + 1, step))
            elif pv_wait(j, "end" if warps[w] + 1 == len(warp) else "behind"):
                moves.append((at, completed, asked, landed, arrived, step))
        if not moves and any(p < len(warp) for p in warps):
            raise Fault(f"nothing can move: issuing thread at {program[at] if at < len(program) else 'its end'}, warps at "
                        f"{[warp[p] if p < len(warp) else 'the end' for p in warps]}")
        for move in moves:
            if move not in seen:
                seen.add(move)
                todo.append(move)
    return len(seen)


@pytest.mark.parametrize("n,ragged", [(1, True), (2, False), (2, True), (3, True), (4, False), (5, True)])
def test_no_order_of_events_passes_a_wait_early_or_stops(header, n, ragged):
    slot, parity = header
    assert walk(n, slot, parity, ragged=ragged) > 10 * n


def test_the_walk_finds_what_one_barrier_for_all_tiles_gets_wrong():
    """The model itself: with one barrier the last wait is passed two products early; warps that follow the products behind
    their own arrival, or an issuing thread that is slow to look at its barrier, can wait for ever."""
    one, two = ((lambda j: 0), (lambda j: j & 1)), ((lambda j: j & 1), (lambda j: j >> 1 & 1))
    with pytest.raises(Fault, match="passed before it was over"):
        walk(2, *one, hand_on=two)
    with pytest.raises(Fault, match="nothing can move"):
        walk(3, *one, hand_on=two, behind=True)
    with pytest.raises(Fault, match="nothing can move"):
        walk(3, *two, hand_on=one)
