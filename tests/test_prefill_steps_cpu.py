"""CPU: the barrier protocol of a query tile in the head_dim 128 / 64 prompt attention (csrc/prefill_tc5.cu), walked through every
order in which the issuer, the tensor pipe and the softmax warps can run: no warp may be left waiting, and no wait for "P.V of step u
is complete" may pass before it is.  The barrier and phase of a step are the kernel's own (csrc/prefill_tc5_steps.h)."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hyprstream_b200", "csrc")
WARPS = 2  # softmax warps of the tile (the kernel has four; two already differ in how far they are)


@pytest.fixture(scope="module")
def kernel_plan(tmp_path_factory):
    """(barrier, parity) of a step as the kernel has them."""
    d = tmp_path_factory.mktemp("steps")
    (d / "s.cpp").write_text('#include "prefill_tc5_steps.h"\nextern "C" int bar(int u) { return hs::t5_odone_bar(u); }\n'
                             'extern "C" int parity(int u) { return static_cast<int>(hs::t5_odone_parity(u)); }\n')
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "s.so"), str(d / "s.cpp")])
    lib = ctypes.CDLL(str(d / "s.so"))
    return lambda u: (lib.bar(u), lib.parity(u))


def explore(nt, plan, epilogue):
    """(left waiting, passed too early) over all orders, for nt steps; `epilogue`: the steps a warp waits for at its end."""
    order = [("S", 0)] + ([("S", 1)] if nt > 1 else [])  # the issuer's operations; they execute, and arrive, in issue order
    for u in range(nt):
        order += [("PV", u)] + ([("S", u + 2)] if u + 2 < nt else [])

    def passes(done, bar, parity, kind):
        phases = sum(1 for k, u in order[:done] if k == kind and (plan(u)[0] if kind == "PV" else u & 1) == bar)
        return (phases & 1) != parity

    # a warp's program: per step see the scores, perhaps (a rescale) wait for the step before, hand over P; then the epilogue
    prog = []
    for u in range(nt):
        prog += [("scores", u)] + ([("rescale", u - 1)] if u else []) + [("P", u)]
    prog += [("done", u) for u in epilogue(nt)]
    start = (0, 0, (0,) * WARPS)  # operations issued, completed, each warp's place in its program
    todo, seen, stuck, early = [start], {start}, False, False
    while todo:
        issued, done, at = todo.pop()
        nxt = []
        if issued < len(order):
            kind, u = order[issued]
            # P.V_u waits for every warp's P_u: its buffer's barrier counts the warps for the u // 2-th time
            if kind == "S" or all(a > prog.index(("P", u)) for a in at):
                nxt.append((issued + 1, done, at))
        if done < issued:
            nxt.append((issued, done + 1, at))
        for w in range(WARPS):
            if at[w] == len(prog):
                continue
            step, u = prog[at[w]]
            ahead = at[:w] + (at[w] + 1,) + at[w + 1:]
            if step == "P" or step == "rescale":  # (a rescale may not be needed)
                nxt.append((issued, done, ahead))
            if step == "scores" and passes(done, u & 1, (u >> 1) & 1, "S"):
                early |= ("S", u) not in order[:done]
                nxt.append((issued, done, ahead))
            if step in ("rescale", "done"):
                if passes(done, *plan(u), "PV"):
                    early |= ("PV", u) not in order[:done]
                    nxt.append((issued, done, ahead))
                else:
                    stuck |= ("PV", u) in order[:done]  # complete, and the wait does not see it
        stuck |= not nxt and not (done == len(order) and all(a == len(prog) for a in at))
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return stuck, early


@pytest.mark.parametrize("nt", range(1, 8))
def test_every_wait_ends_and_none_passes_early(kernel_plan, nt):
    assert explore(nt, kernel_plan, lambda n: [n - 1]) == (False, False)


def test_one_barrier_for_all_steps_would_not_do():
    """... waited for by its last two phases in turn: a warp that looks late waits for a parity that never comes."""
    assert explore(4, lambda u: (0, u & 1), lambda n: [n - 2, n - 1])[0]
