"""Model check of the copies in flight in bcl_b200/csrc/spmm.cu's long-row kernels
(no GPU): the pair of warps of k_spmm_long (spmm_long_row) and the block of
k_spmm_chain (chain_row), each as two actors that meet at barriers.

Between two meetings the actors run in any order, so a slot that one of them
writes there must not be one that the other reads there.  The producers' copies
land in commit groups, oldest first, and are seen by the consumer past a meeting
that follows the wait.  For every number of chunks the models check that what
is read has landed and is the chunk asked for, and that no slot is written
before its last reader is past a meeting.  Fewer slots, or a wait that leaves
one more group in flight, are found."""
import pytest


class Slots:
    """Shared-memory slots: what each holds, whether its copies have landed, and in
    which interval (between two meetings) it was last read by the other actor."""

    def __init__(self, n):
        self.n, self.holds, self.read = n, {}, {}

    def write(self, x, interval):
        s = x % self.n
        assert self.read.get(s, -1) < interval, f"slot {s} written for {x} while it is read"
        old = self.holds.get(s)
        assert old is None or old in self.done, f"slot {s} overwritten for {x} before {old} was used"
        self.holds[s] = x

    done = frozenset()

    def use(self, x, interval, ready):
        s = x % self.n
        assert self.holds.get(s) == x, f"slot {s} holds {self.holds.get(s)}, not {x}"
        assert x in ready, f"{x} is read before its copies have landed"
        self.read[s] = interval
        self.done = self.done | {x}


class Copies:
    def __init__(self):
        self.open, self.groups, self.landed = set(), [], set()

    def add(self, what):
        self.open.add(what)

    def commit(self):
        self.groups.append(self.open)
        self.open = set()

    def wait(self, pending):
        for g in self.groups[:len(self.groups) - pending]:
            self.landed |= g

    def of(self, kind):
        return {x for k, x in self.landed if k == kind}


def long_row_pair(nch, pending=1, aslots=6, bslots=3, tslots=3):
    """Producer: stages A six chunks ahead, builds and copies B two ahead.  Consumer:
    applies chunk c in interval c + 1 (interval 0 is the fill)."""
    cp = Copies()
    a, b, tab = Slots(aslots), Slots(bslots), Slots(tslots)

    def issue_a(x):
        if x < nch:
            a.write(x, 10 ** 9)  # (read by the same warp: only what it holds matters)
            cp.add(("a", x))

    def build(x, interval):
        if x < nch:
            a.use(x, -1, cp.of("a"))
            tab.write(x, interval)

    def issue_b(x, interval):
        if x < nch:
            assert tab.holds[x % tab.n] == x
            b.write(x, interval)
            cp.add(("b", x))

    issue_a(0), issue_a(1), cp.commit(), issue_a(2), issue_a(3), cp.commit()
    cp.wait(1)
    build(0, 0), build(1, 0)
    issue_b(0, 0), issue_a(4), cp.commit(), issue_b(1, 0), issue_a(5), cp.commit()
    cp.wait(pending)
    for c in range(nch):  # interval c + 1
        seen = cp.of("b")  # what the meeting before it showed
        built = set(tab.holds.values())
        # consumer and producer side by side: the reads are noted first
        b.use(c, c + 1, seen)
        tab.use(c, c + 1, built)
        b.done, tab.done = b.done - {c}, tab.done - {c}  # (done for the producer past the next meeting only)
        issue_a(c + 6)
        build(c + 2, c + 1)
        issue_b(c + 2, c + 1)
        cp.commit()
        cp.wait(pending)
        b.done, tab.done = b.done | {c}, tab.done | {c}


def chain_block(nb, pending=1, buffers=3):
    """Producers: batches b + 1 and b + 2 in flight while b is applied; one barrier a
    batch; the A entries of batch b + 3 are in registers.  A batch's values are
    written at once, its slices copied."""
    cp, buf = Copies(), Slots(buffers)
    fetched = []

    def fetch(x):
        fetched.append(x)

    def issue(x, interval):
        assert fetched[-1] == x, "the pending entries are another batch's"
        if x < nb:
            buf.write(x, interval)
            cp.add(("s", x))
        cp.commit()

    fetch(0), issue(0, 0), fetch(1), issue(1, 0), fetch(2)
    for b in range(nb):  # interval b + 1, past barrier b
        cp.wait(pending)
        buf.use(b, b + 1, cp.of("s"))
        buf.done = buf.done - {b}
        issue(b + 2, b + 1)
        fetch(b + 3)
        buf.done = buf.done | {b}


@pytest.mark.parametrize("nch", list(range(1, 41)))
def test_long_row_pair(nch):
    long_row_pair(nch)


@pytest.mark.parametrize("nb", list(range(1, 41)))
def test_chain_block(nb):
    chain_block(nb)


@pytest.mark.parametrize("change", [dict(pending=2), dict(bslots=2), dict(tslots=2), dict(aslots=4)])
def test_a_changed_pair_is_found(change):
    with pytest.raises(AssertionError):
        long_row_pair(20, **change)


@pytest.mark.parametrize("change", [dict(pending=2), dict(buffers=2)])
def test_a_changed_chain_is_found(change):
    with pytest.raises(AssertionError):
        chain_block(20, **change)
