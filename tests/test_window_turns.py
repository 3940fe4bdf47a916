"""Who may store probabilities when, in the two-tile window kernel (attention_prefill_tc.cu, LINES): a model of its barriers on the CPU.

One warp issues all MMAs, which run in that order; two groups of softmax threads take turns with one buffer of scores and one of probabilities.  A
wait knows a phase by its parity alone, so a barrier may never be two phases ahead of who waits for it.  The model runs the roles under random
schedules over the items (runs of list tiles: their steps under windows, chunks and page shares) and finds stalls and probabilities overwritten
before they were multiplied."""
import random

import pytest

KV, ROWS, SHARE_STEPS = 128, 128, 4


def item(p0, positions, rep, window=0, chunk=0, shares=1, z=0):
    """Steps [ja, jb) of the two tiles of a run (pt_run_item), or of share z of them; their number."""
    lo, j = [], []
    for u in (0, 1):
        p, last = p0 + u * ROWS // rep, p0 + min((u + 1) * ROWS // rep, positions) - 1
        first = max(0, p - window + 1) if window else 0
        lo.append(max(first, p // chunk * chunk) if chunk else first)
        j.append(last // KV + 1 if u * ROWS < positions * rep else 0)
    j0 = lo[0] // KV
    J = max(j) - j0
    shares = max(1, min(shares, J // SHARE_STEPS))
    per = (J + shares - 1) // shares
    z0 = min(J, z * per)
    z1 = min(J, z0 + per)
    ja = [max(lo[u] // KV - j0 - z0, 0) for u in (0, 1)]
    return ja, [max(min(j[u] - j0 - z0, z1 - z0), ja[u]) for u in (0, 1)], z1 - z0


class Barrier:
    def __init__(self, count=1):
        self.count, self.left, self.phase = count, count, 0

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left, self.phase = self.count, self.phase + 1

    def passes(self, n):                       # mbarrier.try_wait.parity for phase n: all that the hardware compares
        return (self.phase & 1) != (n & 1)


def stall(items, rule, rng):
    """None, or what went wrong.  rule "turn": the kernel's; "replay": phases of the other tile's o_full waited for one by one."""
    B = {k: [Barrier(), Barrier()] for k in ("q_full", "q_empty", "s_full", "p_full", "o_full", "turn")}
    B["s_empty"] = [Barrier()]
    queue, stored, wrong = [], [], []          # the tensor pipe; probabilities in the buffer

    def issuer():
        n_s, ns, nq = 0, [0, 0], [0, 0]

        def turn(t):
            if n_s:
                queue.append(("turn", t))
            else:
                B["turn"][t].arrive()
        for ja, jb, J in items:
            on = lambda t, j: ja[t] <= j < jb[t]
            if J:
                assert on(0, 0) or on(1, 0)
                turn(0 if on(0, 0) else 1)
            order = [("s", 0, 0), ("s", 1, 0), ("s", 0, 1)] + [op for j in range(J) for op in (("o", 0, j), ("s", 1, j + 1), ("o", 1, j), ("s", 0, j + 2))]
            for what, t, j in order:
                if not on(t, j):
                    continue
                if what == "s":
                    if j == ja[t]:
                        yield "q_full", t, nq[t]
                        nq[t] += 1
                    if n_s:
                        yield "s_empty", 0, n_s - 1
                    n_s += 1
                    queue.append(("s_full", t))
                    if j + 1 == jb[t]:
                        queue.append(("q_empty", t))
                else:
                    yield "p_full", t, ns[t]
                    ns[t] += 1
                    queue.append(("pv", t))
                    after = [u for u, k in ((1, j) if t == 0 else (0, j + 1), (0, j + 1), (1, j + 1)) if on(u, k)]
                    if after:
                        turn(after[0])
                    if rule == "replay" or j + 1 == jb[t]:
                        queue.append(("o_full", t))

    def softmax(t):
        ns = nq = no = other = seen = 0

        def load(of):
            nonlocal nq
            if of[1][t] > of[0][t]:
                if nq:
                    yield "q_empty", t, nq - 1
                nq += 1
                B["q_full"][t].arrive()
        if items:
            yield from load(items[0])
        for i, (ja, jb, J) in enumerate(items):
            for j in range(ja[t], jb[t]):
                yield "s_full", t, ns
                yield "work", t, 0
                B["s_empty"][0].arrive()
                yield "work", t, 0
                if rule == "turn":
                    yield "turn", t, ns
                else:
                    if j > ja[t]:
                        yield "o_full", t, ns - 1
                    up_to = other + max(0, min(j + t, jb[t ^ 1]) - ja[t ^ 1])
                    while seen != up_to:
                        yield "o_full", t ^ 1, seen
                        seen += 1
                if stored:
                    wrong.append("probabilities overwritten")
                stored.append(t)
                B["p_full"][t].arrive()
                ns += 1
            other += jb[t ^ 1] - ja[t ^ 1]
            if i + 1 < len(items):
                yield from load(items[i + 1])
            if jb[t] > ja[t]:
                yield "o_full", t, (no if rule == "turn" else ns - 1)
                no += 1

    roles = [issuer(), softmax(0), softmax(1)]
    weight = [rng.choice([1, 1, 8]) for _ in range(4)]
    waits = [next(r, None) for r in roles]
    while any(w is not None for w in waits):
        able = [i for i, w in enumerate(waits) if w is not None and (w[0] == "work" or B[w[0]][w[1]].passes(w[2]))]
        if queue:
            able.append(3)
        if not able:
            return f"all wait: {waits}"
        i = rng.choices(able, [weight[k] for k in able])[0]
        if i < 3:
            waits[i] = next(roles[i], None)
            continue
        what, t = queue.pop(0)
        if what != "pv":
            B[what][t].arrive()
        elif stored != [t]:
            return f"P V of tile {t} with the probabilities of {stored}"
        else:
            stored.clear()
        if wrong:
            return wrong[0]
    return None


PLAIN = [[item(0, 64, 4)], [item(64 * k, 64, 4, window=1024) for k in (20,)]]
GEOMETRIES = [
    [item(256, 16, 4), item(0, 48, 4)],                                    # the last tile of one prompt and three of the next
    [item(512 - 32, 48, 4), item(0, 16, 4)],                               # the second tile sees a step more, and another run follows
    [item(2048 - 32, 64, 4, chunk=1024)],                                  # a chunk's border between the tiles
    [item(2000, 64, 4, window=1024, chunk=512), item(0, 16, 4)],
    [item(1007, 64, 4, window=256)],                                  # a window that starts a step later for the second tile
    [item(300, 16, 4), item(700, 16, 4), item(40, 16, 4), item(2000, 16, 4)],
    [item(p0, n, rep, window=w) for p0, n, rep, w in ((900, 7, 8, 0), (300, 24, 8, 256))],
]
GEOMETRIES += [[item(4000, 64, 4, window=w, shares=4, z=z)] for w in (0, 2000) for z in range(4)]


@pytest.mark.parametrize("items", PLAIN + GEOMETRIES)
def test_probabilities_take_turns(items):
    for seed in range(100):
        assert stall(items, "turn", random.Random(seed)) is None


def test_probabilities_take_turns_at_random():
    """Runs as prompts of any lengths behind any histories cut them."""
    rng = random.Random(1)
    for _ in range(1000):
        rep = rng.choice([1, 2, 4, 8, 16, 32, 64])
        rq, window, chunk, shares = 64 // rep, rng.choice([0, 0, 100, 256, 1000, 1024]), rng.choice([0, 0, 0, 512, 1024]), rng.choice([1, 1, 1, 3, 8])
        tiles, items, z = 4, [], rng.randrange(shares)
        while tiles:
            k = rng.randint(1, tiles)
            items.append(item(rng.randrange(3000), rng.randint((k - 1) * rq + 1, k * rq), rep, window, chunk, shares, z))
            tiles -= k
        assert stall(items, "turn", rng) is None, items


@pytest.mark.parametrize("items", GEOMETRIES[:5])
def test_the_model_finds_a_phase_that_passed(items):
    """Waits for the other tile's phases one by one: its barrier may be two of them ahead, where the parity is the one of before."""
    assert any(stall(items, "replay", random.Random(seed)) for seed in range(20))
