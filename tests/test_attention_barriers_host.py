"""The barriers between the roles of the attention backward's dK/dV kernel, as a model on the CPU.

A wait on an mbarrier names a phase by its parity: it passes while the phase in progress has the other parity.  It
therefore means what it says only if the barrier can be neither one phase behind nor one phase ahead of what the waiting
role expects.  The model steps the roles in every order there is and checks both, and that nobody waits for ever."""
import os
import re

import pytest

from conftest import CSRC


def kernel_constant(name):
    with open(os.path.join(CSRC, "attention.cu")) as f:
        return int(re.search(r"constexpr int %s = (\d+);" % name, f.read()).group(1))


def programs(items, ds_free, float_outputs):
    """The waits (barrier, phase) and arrivals (barrier,) of each role, for items of the given numbers of blocks."""
    compute, issuer, store = [], [], [("w_free",)]
    g = 0
    for k, blocks in enumerate(items):
        for it in range(blocks):
            compute.append(("w_free", g - 1))                # (block 0: the phase before the first, which passes)
            if it == 0 and k > 0:
                compute.append(("out_done", k - 1))
            compute.append(("pds_full",))
            issuer += [("pds_full", g), ("w_free",), ("ds_free%d" % (g % ds_free),)]
            store += [("ds_free%d" % (g % ds_free), g // ds_free), ("w_free",)]
            g += 1
        issuer.append(("acc_full",))
        compute.append(("acc_full", k))
        if float_outputs:
            compute.append(("w_free", g - 1))
        compute.append(("out_full",))
        store += [("out_full", k), ("out_done",)]
    return [compute, issuer, store]


def explore(items, ds_free, float_outputs):
    """None, or what can go wrong."""
    prog = programs(items, ds_free, float_outputs)
    needed = {"w_free": 2}
    start = (0, 0, 0)
    seen, todo = {start}, [start]
    while todo:
        at = todo.pop()
        arrived = {}
        for p, n in zip(prog, at):
            for op in p[:n]:
                if len(op) == 1:
                    arrived[op[0]] = arrived.get(op[0], 0) + 1
        moved = False
        for r in range(3):
            if at[r] == len(prog[r]):
                continue
            op = prog[r][at[r]]
            if len(op) == 2:
                completed = arrived.get(op[0], 0) // needed.get(op[0], 1)
                if (completed & 1) == (op[1] & 1):           # the phase in progress has the parity that is waited for
                    continue
                if completed <= op[1]:
                    return "%s: phase %d taken for complete after %d" % (op[0], op[1], completed)
            moved = True
            nxt = at[:r] + (at[r] + 1,) + at[r + 1:]
            if nxt not in seen:
                seen.add(nxt)
                todo.append(nxt)
        if not moved and any(n < len(p) for n, p in zip(at, prog)):
            return "nobody can go on at %r" % [p[n] if n < len(p) else "end" for n, p in zip(at, prog)]
    return None


@pytest.mark.parametrize("float_outputs", [False, True])
@pytest.mark.parametrize("items", [(1,), (4,), (1, 1, 1), (2, 1, 3), (3, 3, 2), (1, 4, 1, 2)])
def test_no_order_of_the_roles_loses_a_phase(items, float_outputs):
    assert explore(items, kernel_constant("ATT_DS_FREE"), float_outputs) is None


def test_the_model_sees_a_barrier_that_can_run_ahead():
    """With one barrier for all blocks the store thread can be two phases late."""
    assert "nobody can go on" in explore((3, 3, 2), 1, False)
