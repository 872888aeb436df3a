"""The roles of the attention backward kernel over several items of one CTA (blocks of 128 keys, one after the other), at any
speed relative to each other.  Steps of a block are read from the source; what lies between two items stands here."""
import pytest

from tests.test_kernel_contracts_cpu import STAGES, _bwd_roles


def _programs(nq, items):
    """{actor: [step]}; products and the commits behind them are steps of a queue that the tensor core works off.  `data`:
    what a place holds, (name, place) -> block or item."""
    total = nq * items
    roles = _bwd_roles()
    P = {a: [] for a in ("load", "grad", "drain", "math", "load queue", "grad queue")}

    def wait(role, name, index, phase):
        P[role].append(("wait", (name, index), phase))

    def arrive(role, name, index=0):
        P[role].append(("arrive", (name, index)))

    def queue(role, step):
        P[role + " queue"].append((*step, len(P[role])))

    def put(role, bar, place, what):
        P[role].append(("put", bar, place, what))

    # ---- load warp
    put("load", ("kv_full", 0), ("K", 0), 0)
    put("load", None, ("V", 0), 0)
    for c in range(min(STAGES, total)):
        put("load", ("qd_full", c % STAGES), ("Q", c % STAGES), c)
    for k in range(items):
        wait("load", "kv_full", 0, k)
        for i in range(nq):
            c = k * nq + i
            assert [n for w, n in roles["load"] if w != "C_"] == ["qd_full", "s_free", "s_full", "qd_free", "i"]
            wait("load", "qd_full", c % STAGES, c // STAGES)
            if c > 0:
                wait("load", "s_free", 0, c - 1)
            queue("load", ("read", [(("K", k & 1), k), (("Q", c % STAGES), c), (("V", 0), k)]))
            queue("load", ("arrive", ("s_full", 0)))
            if i + 1 < nq and c >= 1 and c + 2 < total:
                wait("load", "qd_free", (c + 2) % STAGES, (c - 1) // STAGES)
                put("load", ("qd_full", (c + 2) % STAGES), ("Q", (c + 2) % STAGES), c + 2)
        c = (k + 1) * nq - 1
        if k + 1 < items:
            wait("load", "s_full", 0, c)
            if k > 0:
                wait("load", "k_free", (k + 1) & 1, (k - 1) >> 1)
            put("load", ("kv_full", 0), ("K", (k + 1) & 1), k + 1)
            put("load", None, ("V", 0), k + 1)
        if c >= 1 and c + 2 < total:
            wait("load", "qd_free", (c + 2) % STAGES, (c - 1) // STAGES)
            put("load", ("qd_full", (c + 2) % STAGES), ("Q", (c + 2) % STAGES), c + 2)
    # ---- gradient products
    for k in range(items):
        if k > 0:
            wait("grad", "dkv_taken", 0, k - 1)
        for i in range(nq):
            c = k * nq + i
            wait("grad", "qd_full", c % STAGES, c // STAGES)
            wait("grad", "pds_ready", 0, c)
            queue("grad", ("read", [(("Q", c % STAGES), c), (("K", k & 1), k), (("dS", 0), c), (("P", 0), c)]))
            if c > 0:
                wait("grad", "dq_taken", 0, c - 1)
            queue("grad", ("arrive", ("ds_done", 0)))
            if c + STAGES < total:
                queue("grad", ("arrive", ("qd_free", c % STAGES)))
            queue("grad", ("arrive", ("p_done", 0)))
        if k + 2 < items:
            queue("grad", ("arrive", ("k_free", k & 1)))
    # ---- drain
    for c in range(min(2, total)):
        arrive("drain", "stats_full", c & 1)
    for k in range(items):
        for i in range(nq):
            c = k * nq + i
            wait("drain", "ds_done", 0, c)
            arrive("drain", "dq_taken")
            if c + 2 < total:
                arrive("drain", "stats_full", c & 1)
        wait("drain", "p_done", 0, (k + 1) * nq - 1)
        arrive("drain", "dkv_taken")
    # ---- math
    for c in range(total):
        wait("math", "stats_full", c & 1, c >> 1)
        wait("math", "s_full", 0, c)
        arrive("math", "s_free")
        if c > 0:
            wait("math", "ds_done", 0, c - 1)
        P["math"].append(("put", None, ("dS", 0), c))
        if c > 0:
            wait("math", "p_done", 0, c - 1)
        P["math"].append(("put", None, ("P", 0), c))
        arrive("math", "pds_ready")
    return P


@pytest.mark.parametrize("nq,items", [(1, 1), (1, 2), (1, 5), (2, 3), (3, 3), (4, 2), (5, 2)])
def test_roles_over_several_items_at_any_speed(nq, items):
    progs = _programs(nq, items)
    actors = list(progs)
    arrived = {a: [{}] for a in actors}
    held = {a: [{}] for a in ("load", "math")}
    for a in actors:
        for step in progs[a]:
            count = dict(arrived[a][-1])
            if step[0] == "arrive":
                count[step[1]] = count.get(step[1], 0) + 1
            if step[0] == "put" and step[1]:
                count[step[1]] = count.get(step[1], 0) + 1
            if a in held:
                held[a].append({**held[a][-1], step[2]: step[3]} if step[0] == "put" else held[a][-1])
            arrived[a].append(count)

    def ended(bar, at):
        return sum(arrived[a][pc].get(bar, 0) for a, pc in zip(actors, at))

    seen, todo = set(), [(0,) * len(actors)]
    while todo:
        at = todo.pop()
        if at in seen:
            continue
        seen.add(at)
        moves = 0
        for k, a in enumerate(actors):
            if at[k] == len(progs[a]):
                continue
            step = progs[a][at[k]]
            if step[0] == "wait":
                n = ended(step[1], at)
                if (n - step[2]) % 2 == 0:
                    continue
                assert n == step[2] + 1, f"{a} passes {step} with {n} phases ended"
            elif a.endswith("queue"):
                if at[actors.index(a.split()[0])] < step[-1]:
                    continue   # not issued yet
                if step[0] == "read":
                    for place, what in step[1]:
                        owner = "math" if place[0] in ("dS", "P") else "load"
                        assert held[owner][at[actors.index(owner)]].get(place) == what, f"{a}: {place} holds another's"
            moves += 1
            todo.append(at[:k] + (at[k] + 1,) + at[k + 1:])
        assert moves or all(pc == len(progs[a]) for a, pc in zip(actors, at)), \
            "stuck before " + ", ".join(str(progs[a][pc]) for a, pc in zip(actors, at) if pc < len(progs[a]))
