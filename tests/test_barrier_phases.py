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


def stuck(program, two):
    """A reachable state in which somebody waits for a phase that has gone by, or passes one that has not come."""
    issuer, warp = program(two)
    commits = [op[1] for op in issuer if op[0] == "issue"]

    def phase(bar, ws, done):
        arrived = sum(op == ("arrive", bar) for w in ws for op in warp[:w])
        return arrived // 2 + sum(c.count(bar) for c in commits[:done])

    seen, todo = set(), [(0, (0, 0), 0)]
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        ip, ws, done = state
        if done < sum(op[0] == "issue" for op in issuer[:ip]):
            todo.append((ip, ws, done + 1))
        for who, ops, at in [(-1, issuer, ip), (0, warp, ws[0]), (1, warp, ws[1])]:
            if at == len(ops):
                continue
            op = ops[at]
            if op[0] == "wait":
                now = phase(op[1], ws, done)
                if not now - op[2] in (0, 1):
                    return state
                if now == op[2]:
                    continue
            # bar.sync of the compute warps: both have to be there, or the other one is past it
            if op[0] == "meet" and ws[1 - who] < at:
                continue
            todo.append((ip + 1, ws, done) if who < 0 else (ip, tuple(w + (k == who) for k, w in enumerate(ws)), done))
    return None


@pytest.mark.parametrize("program", [fp32_forward, fp32_dkdv, fp32_dq, bwd_dkdv_64, bwd_dkdv_128, bwd_dq])
def test_no_wait_is_overtaken(program):
    assert stuck(program, True) is None


@pytest.mark.parametrize("program", [fp32_forward, bwd_dkdv_64])
def test_one_barrier_for_p_is_overtaken_where_scores_run_ahead(program):
    assert stuck(program, False) is not None
