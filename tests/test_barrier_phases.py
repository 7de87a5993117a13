"""Hand-shakes between the MMA issuer and the compute warps of the attention kernels, every interleaving of two compute warps.

A wait by parity passes when the barrier's current phase has the other parity.  It is sound only while the barrier is at the
waiter's phase or one further: two further, and the wait for a phase that is long over blocks until it gives up.  The programs
below are the waits, arrivals and commits of the kernels, step by step; products complete in the order in which they are
issued, any time later."""
import pytest

N = 5


def fp32_forward(two):                     # attn_f32.cu, A_FWD: scores two steps ahead of P
    p = lambda i: (("p", i & 1), i >> 1) if two else (("p", 0), i)
    issuer = [("issue", [("s", i)]) for i in (0, 1)]
    warp = []
    for i in range(N):
        issuer += [("wait", *p(i)), ("issue", [("acc", i & 1)])]
        issuer += [("issue", [("s", i & 1)])] if i + 2 < N else []
        warp += [("wait", ("s", i & 1), i >> 1), ("meet",), ("arrive", p(i)[0])]
        warp += [("wait", ("acc", (i - 1) & 1), (i - 1) >> 1)] if i else []
    return issuer, warp + [("wait", ("acc", (N - 1) & 1), (N - 1) >> 1)]


def fp32_dkdv(two):                        # A_DKDV: S of the next step follows P of this one
    issuer, warp = [("issue", [("s", 0)]), ("issue", [("dp", 0)])], []
    for i in range(N):
        more = i + 1 < N
        issuer += [("wait", ("p", 0), i), ("issue", [])] + ([("issue", [("s", 0)])] if more else [])
        issuer += [("wait", ("ds", 0), i), ("issue", [])] + [("issue", [("dp", 0)] if more else [("acc", 0)])]
        warp += [("wait", ("s", 0), i), ("arrive", ("p", 0)), ("wait", ("dp", 0), i), ("arrive", ("ds", 0))]
    return issuer, warp + [("wait", ("acc", 0), 0)]


def fp32_dq(two):                          # A_DQ: S one step ahead, in the other of two regions
    issuer, warp = [("issue", [("s", 0)]), ("issue", [("dp", 0)])], []
    for i in range(N):
        more = i + 1 < N
        issuer += ([("issue", [("s", (i + 1) & 1)])] if more else []) + [("wait", ("ds", 0), i), ("issue", [])]
        issuer += [("issue", [("dp", 0)] if more else [("acc", 0)])]
        warp += [("wait", ("s", i & 1), i >> 1), ("wait", ("dp", 0), i), ("arrive", ("ds", 0))]
    return issuer, warp + [("wait", ("acc", 0), 0)]


def bwd_dkdv(scores, two):                 # flash_bwd_sm100.cu: `scores` buffers of S, as many query tiles ahead
    s = lambda i: (("s", i % scores), i // scores)
    p = lambda i: (("p", i & 1), i >> 1) if two and scores == 2 else (("p", 0), i)
    issuer, warp = [("issue", [s(0)[0]]), ("issue", [("dp", 0)])] + ([("issue", [s(1)[0]])] if scores == 2 else []), []
    for i in range(N):
        issuer += [("wait", *p(i)), ("issue", [])] + ([("issue", [s(i + scores)[0]])] if i + scores < N else [])
        issuer += [("wait", ("ds", 0), i), ("issue", [])] + ([("issue", [("dp", 0)])] if i + 1 < N else [])
        # (row vectors; columns read before they are written over)
        warp += [("meet",), ("wait", *s(i)), ("meet",), ("arrive", p(i)[0]), ("wait", ("dp", 0), i), ("meet",), ("arrive", ("ds", 0))]
    return issuer + [("issue", [("acc", 0)])], warp + [("wait", ("acc", 0), 0)]


def bwd_dkdv_64(two):
    return bwd_dkdv(2, two)


def bwd_dkdv_128(two):
    return bwd_dkdv(1, two)


def bwd_dq(two):                           # S up to two key tiles ahead, dP one
    issuer, warp = [("issue", [("s", 0)]), ("issue", [("dp", 0)]), ("issue", [("s", 1)])], []
    for i in range(N):
        issuer += [("wait", ("ds", 0), i), ("issue", [])] + ([("issue", [("dp", 0)])] if i + 1 < N else [])
        issuer += [("issue", [("s", i & 1)])] if i + 2 < N else []
        warp += [("wait", ("s", i & 1), i >> 1), ("wait", ("dp", 0), i), ("meet",), ("arrive", ("ds", 0))]
    return issuer + [("issue", [("acc", 0)])], warp + [("wait", ("acc", 0), 0)]


def forward_queue(s_own, o_own, nbuf=3, items=((1, 2), (3, 0), (3, 0), (1, 2))):
    """flash_fwd_sm100.cu, persistent: key tiles of the two query tiles of each item, longest first in a group, so that items
    without a second tile follow those of the group before.  s_own: score barriers of each query tile's own, four in turn; o_own:
    a barrier of its own behind the last product of a query tile."""
    sched, scores, outs, warps = [], [], [], ([], [])
    gs, taken, done, before = 0, [0, 0], [0, 0], [None, None]
    for n, nk in enumerate(items):
        sched += ([("wait", ("w_empty", n & 1), n // 2 - 1)] if n > 1 else []) + [("arrive", ("w_full", n & 1))]
        for a in (scores, outs, *warps):
            a += [("wait", ("w_full", n & 1), n // 2), ("arrive", ("w_empty", n & 1))]
        order = [(t, j) for j in range(nk[0]) for t in ((0, 1) if nk[1] else (0,))] + [(1, j) for j in range(nk[0], nk[1])]
        for t, j in order:
            buf, k = gs % nbuf, gs // nbuf
            s = (("s", t, taken[t] & 3), taken[t] >> 2) if s_own else (("s", buf), k)
            scores += ([("wait", ("free", buf), k - 1)] if k else []) + [("issue", [s[0]])]
            last = j == nk[t] - 1
            outs += [("wait", ("o_free", t), done[t] - 1)] if j == 0 and done[t] else []
            outs += [("wait", ("p", buf), k), ("issue", [("free", buf)] + ([("o", t)] if last else []))]
            # (a larger row maximum rescales O, once the product of the step before is done)
            warps[t].extend([("wait", *s)] + ([("wait", ("free", before[t][0]), before[t][1])] if j else []) + [("arrive", ("p", buf))])
            before[t] = buf, k
            if last:
                warps[t].extend([("wait", ("o", t), done[t]) if o_own else ("wait", ("free", buf), k), ("arrive", ("o_free", t))])
                done[t] += 1
            taken[t] += 1
            gs += 1
    return [sched, scores, outs, *warps], {"w_empty": 4}


def stuck(agents, counts):
    """A reachable state in which somebody waits for a phase that has gone by, or passes one that has not come.  counts: arrivals
    that make a phase, by the barrier's name, where it is not one; the agents that meet are the ones with such an operation."""
    commits = [[op[1] for op in a if op[0] == "issue"] for a in agents]
    bars = {op[1] for a in agents for op in a if op[0] in ("wait", "arrive")}
    arrived = {b: [[sum(op == ("arrive", b) for op in a[:n]) for n in range(len(a) + 1)] for a in agents] for b in bars}
    committed = {b: [[sum(x.count(b) for x in c[:n]) for n in range(len(c) + 1)] for c in commits] for b in bars}
    issued = [[sum(op[0] == "issue" for op in a[:n]) for n in range(len(a) + 1)] for a in agents]

    def phase(b, at, done):
        return (sum(arrived[b][i][n] for i, n in enumerate(at)) // counts.get(b[0], 1)
                + sum(committed[b][i][n] for i, n in enumerate(done)))

    seen, todo = set(), [((0,) * len(agents), (0,) * len(agents))]
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        at, done = state
        for i, ops in enumerate(agents):
            if done[i] < issued[i][at[i]]:
                todo.append((at, done[:i] + (done[i] + 1,) + done[i + 1:]))
            if at[i] == len(ops):
                continue
            op = ops[at[i]]
            if op[0] == "wait":
                now = phase(op[1], at, done)
                if not now - op[2] in (0, 1):
                    return state
                if now == op[2]:
                    continue
            # bar.sync: everybody is there, or past it
            if op[0] == "meet" and any(at[k] < at[i] for k, a in enumerate(agents) if ("meet",) in a):
                continue
            todo.append((at[:i] + (at[i] + 1,) + at[i + 1:], done))
    return None


def two_warps(program, two):
    issuer, warp = program(two)
    return [issuer, warp, warp], {"p": 2, "ds": 2}


@pytest.mark.parametrize("program", [fp32_forward, fp32_dkdv, fp32_dq, bwd_dkdv_64, bwd_dkdv_128, bwd_dq])
def test_no_wait_is_overtaken(program):
    assert stuck(*two_warps(program, True)) is None


@pytest.mark.parametrize("program", [fp32_forward, bwd_dkdv_64])
def test_one_barrier_for_p_is_overtaken_where_scores_run_ahead(program):
    assert stuck(*two_warps(program, False)) is not None


@pytest.mark.parametrize("nbuf", [2, 3])
def test_forward_queue(nbuf):
    assert stuck(*forward_queue(True, True, nbuf)) is None
    assert stuck(*forward_queue(False, True, nbuf)) is not None
    assert stuck(*forward_queue(True, False, nbuf)) is not None
