"""The roles of the attention backward kernel over several items of one CTA (blocks of 128 keys, one after the other), at any
speed relative to each other.  The programs stand here; the operations they are made of are compared with the source."""
import pytest

from tests.test_kernel_contracts_cpu import STAGES, TOKEN, _closing, _kernels

# A role's barrier operations, products and loads in the order of the source, over a block and between items
SOURCE = {
    "load": "wait kv_full, wait qd_full, wait s_free, C_ ST, C_ DPT, commit s_full, wait qd_free, load_qd i, wait s_full, "
            "wait k_free, wait qd_free",
    "grad": "wait dkv_taken, wait qd_full, wait pds_ready, C_ DK, wait dq_taken, C_ DQ, commit ds_done, C_ DV, commit qd_free, "
            "commit p_done, commit k_free",
    "drain": "arrive stats_full, wait ds_done, arrive dq_taken, put_stats i, arrive dq_free, wait dq_free, arrive dq_ready, "
             "wait dq_ready, wait p_done, arrive dkv_taken, arrive dkv_free, wait dkv_free, arrive dkv_ready, wait dkv_ready",
    "math": "wait stats_full, wait s_full, arrive s_free, wait ds_done, wait p_done, arrive pds_ready",
}
# the drain's first warp issues the copies; the others are the second actor, and barriers count both
BOTH = ("dq_taken", "dkv_taken", "stats_full", "dq_ready", "dkv_ready")


def test_operations_of_the_roles_are_those_of_the_source():
    body = _kernels("attn_bwd.cu")["attn_bwd_kernel"][1]
    start = body.index("if (warp == LOAD_WARP) {", body.index("grid_wait()"))
    for role, want in SOURCE.items():
        open_ = body.index("{", start)
        section = body[open_:_closing(body, open_)]
        start = open_ + len(section)
        assert ", ".join(" ".join(x for x in m.groups() if x) for m in TOKEN.finditer(section)) == want, role
        if role == "drain":
            # every write to the staging memory behind the copies that read it, every copy behind the writes
            assert section.count("tma_store_wait_read<0>()") == 3
            for bar in ("dq", "dkv"):
                at = [section.index(f"mbar_arrive({bar}_free)"), section.index(f"mbar_wait_warp({bar}_free"),
                      section.index(f"mbar_arrive({bar}_ready)"), section.index(f"mbar_wait_warp({bar}_ready")]
                assert at == sorted(at)
                assert section.rindex("tma_store_wait_read<0>()", 0, at[0]) > at[0] - 200
                assert "fence_proxy_async()" in section[at[1]:at[2]]


def _programs(nq, items):
    """{actor: [step]}; products and the commits behind them are steps of a queue that the tensor core works off, the copies
    out of the staging memory of one that the copy engine does.  A place holds a block or an item."""
    total = nq * items
    P = {a: [] for a in ("load", "grad", "drain", "drain 2", "math", "load queue", "grad queue", "drain queue")}

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
    def staged(bar, c, places, what):
        """Both halves of the drain write `what` to a place each, and the first warp has the copy engine read them."""
        if bar:
            P["drain"].append(("drained", len(P["drain queue"])))
            arrive("drain", bar + "_free")
        for h, role in enumerate(("drain", "drain 2")):
            if bar:
                wait(role, bar + "_free", 0, c)
            P[role].append(("put", None, places[h], what))
            arrive(role, ("dkv" if what[0] == "dkv" else "dq") + "_ready")
        wait("drain", ("dkv" if what[0] == "dkv" else "dq") + "_ready", 0, what[1])
        queue("drain", ("read", [(places[0], what), (places[1], what)]))

    def both(name, index=0):
        arrive("drain", name, index)
        arrive("drain 2", name, index)

    for c in range(min(2, total)):
        both("stats_full", c & 1)
    for k in range(items):
        for i in range(nq):
            c = k * nq + i
            for role in ("drain", "drain 2"):
                wait(role, "ds_done", 0, c)
            both("dq_taken")
            if c + 2 < total:
                both("stats_full", c & 1)
            staged("dq", c, (("T", 0), ("T", 1)), ("dq", c))
        for role in ("drain", "drain 2"):
            wait(role, "p_done", 0, (k + 1) * nq - 1)
        both("dkv_taken")
        # (the last item's go where nothing is loaded any more: each half of the drain writes to both, here to one)
        last = k + 1 == items
        staged(None if last else "dkv", k, (("K", (k + 1) & 1), ("V", 0)) if last else (("T", 0), ("T", 1)), ("dkv", k))
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
    held = {a: [{}] for a in ("load", "math", "drain", "drain 2")}
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
        if bar[0] in BOTH:
            n = [arrived[a][at[actors.index(a)]].get(bar, 0) for a in ("drain", "drain 2")]
            assert abs(n[0] - n[1]) <= 1, f"{bar} counts one actor twice"
            return min(n)
        return sum(arrived[a][pc].get(bar, 0) for a, pc in zip(actors, at))

    def holds(owner, place, at):
        return held[owner][at[actors.index(owner)]].get(place)

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
            elif step[0] == "drained":
                if at[actors.index("drain queue")] < step[1]:
                    continue   # a copy still reads
            elif a.endswith("queue"):
                if at[actors.index(a.split()[0])] < step[-1]:
                    continue   # not issued yet
                if step[0] == "read":
                    for h, (place, what) in enumerate(step[1]):
                        drains = ("drain", "drain 2")
                        owner = drains[h] if a == "drain queue" else "math" if place[0] in ("dS", "P") else "load"
                        assert holds(owner, place, at) == what, f"{a}: {place} holds another's"
                        # (K and V have two writers: what the products read has not been written over by the drain)
                        assert owner != "load" or all(holds(d, place, at) is None for d in drains), f"{a}: {place} is gone"
            moves += 1
            todo.append(at[:k] + (at[k] + 1,) + at[k + 1:])
        assert moves or all(pc == len(progs[a]) for a, pc in zip(actors, at)), \
            "stuck before " + ", ".join(str(progs[a][pc]) for a, pc in zip(actors, at) if pc < len(progs[a]))
