"""The four warps of the ragged forward (rope_split_fwd_sm100.cu) that hold the same 32 rows meet at a hardware barrier several times per item.
Between these meetings they wait, with a limit, for TMA loads and MMAs, and any such wait may give up in one warp and not in another.
A model of their program goes through every order of steps and every outcome of every wait: whatever gives up where, all four must end.
(On a GPU this can only be read: a warp that is left alone at the barrier never ends.)"""

import pytest

WARPS, ITEMS, BLOCKS = 4, 2, 2


def carried():
    """The kernel's program: (operation, jump target) where `ok` of a warp that gave up is carried to the next place where all four look."""
    code, leave = [], []

    def look(op):
        code.append([op, None])
        leave.append(len(code) - 1)

    for item in range(ITEMS + 1):                  # the last one is "no item left"
        code += [["wait", None], ["tell_item", None], ["sync", None]]
        if item == ITEMS:
            break
        look("leave_if_told_item")
        code.append(["sync", None])                # the parts of Q
        for block in range(BLOCKS):
            code += [["wait", None], ["tell_block", None], ["sync", None], ["look_block", None]]
            if block > 0:
                code.append(["wait", None])        # the product of the block before
            code.append(["sync", None])
            look("leave_if_told_block")
        code += [["wait", None], ["sync", None], ["sync", None]]
    for at in leave:
        code[at][1] = len(code)
    return code


def alone():
    """A warp that gives up leaves at once and arrives eight times for what may still come."""
    code = []
    for item in range(ITEMS + 1):
        code.append(["wait_or_quit", None])
        if item == ITEMS:
            break
        code.append(["sync", None])
        for block in range(BLOCKS):
            code += [["wait_or_quit", None], ["sync", None]] + ([["wait_or_quit", None]] if block > 0 else []) + [["sync", None]]
        code += [["wait_or_quit", None], ["sync", None], ["sync", None]]
    end = len(code) + 1 + 8
    code.append(["end", end])
    for op in code:
        if op[0] == "wait_or_quit":
            op[1] = len(code)
    return code + [["arrive", None]] * 8


def hangs(code):
    """True if some order of steps ends with a warp at the barrier that nobody will come to."""
    # per warp: (pc, ok, tells the others of this block, was told, at the barrier); shared: told_item, arrivals in the barrier's phase
    start = (((0, True, False, False, False),) * WARPS, False, 0)
    seen, todo = {start}, [start]
    while todo:
        warps, told_item, count = todo.pop()
        moved = False

        def go(i, pc, ok, tells, told, waiting=False, item=told_item, arrivals=count, release=False):
            now = [(w[0] + 1,) + w[1:4] + (False,) if release and w[4] else w for w in warps]
            now[i] = (pc, ok, tells, told, waiting)
            state = (tuple(sorted(now)), item, 0 if release else arrivals)   # the warps are alike
            if state not in seen:
                seen.add(state)
                todo.append(state)

        for i, (pc, ok, tells, told, waiting) in enumerate(warps):
            if waiting or pc >= len(code):
                continue
            moved = True
            op, target = code[pc]
            if op == "wait":
                go(i, pc + 1, ok, tells, told)
                if ok:
                    go(i, pc + 1, False, tells, told)
            elif op == "wait_or_quit":
                go(i, pc + 1, ok, tells, told)
                go(i, target, False, tells, told)
            elif op == "tell_item":
                go(i, pc + 1, ok, tells, told, item=told_item or not ok)
            elif op == "tell_block":
                go(i, pc + 1, ok, not ok, told)
            elif op == "look_block":
                go(i, pc + 1, ok, tells, any(w[2] for w in warps))
            elif op == "leave_if_told_item":
                go(i, target if told_item else pc + 1, ok, tells, told)
            elif op == "leave_if_told_block":
                go(i, target if told else pc + 1, ok, tells, told)
            elif op in ("sync", "arrive"):
                last = count + 1 == WARPS
                go(i, pc + 1 if last or op == "arrive" else pc, ok, tells, told, waiting=op == "sync" and not last, arrivals=count + 1, release=last)
            elif op == "end":
                go(i, target, ok, tells, told)
        if not moved and any(w[4] for w in warps):
            return True
    return False


def test_all_four_warps_end_whichever_wait_gives_up():
    assert not hangs(carried())


def test_the_model_finds_the_warp_that_is_left_alone():
    assert hangs(alone())
