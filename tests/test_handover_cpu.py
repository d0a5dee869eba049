"""Hand-overs of the kernels, walked through exhaustively: every interleaving of small models that have the kernels' waits and
arrivals.  Barriers behave as mbarriers do: a phase ends with the last expected arrival, and a wait sees only the parity of the
phase.  How many barriers a hand-over has is read from the kernels' source.

dS in the dQ kernel (bwd_dq_kernel, csrc/bwd_sm100.cu), one long item: two elementwise warps, the thread that issues S and dP, the
one that issues dQ, and the tensor pipe, which completes each thread's products in order and as late as it likes.

The zeroed tail of V in the forward (fwd_kernel, csrc/fwd_sm100.cu), short items that all need it: the producer warp, the thread that
issues the products, and the tensor pipe.
"""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "flash_attention_turing_b200" / "csrc"
WARPS = 2
BLOCKS = 6
ITEMS = 6


def _barriers(source, struct, name):
    fields = re.search(rf"struct {struct} \{{(.*?)\n\}};", (CSRC / source).read_text(), re.S).group(1)
    several = re.search(rf"\b{name}\[(\d+)\]", fields)
    return int(several.group(1)) if several else 1


class _Fault(Exception):
    pass


def _walk_dq(n_ds):
    """Visits all states; raises _Fault for a product on a packed-dS buffer that is not whole, or for a state without a way on."""
    # barriers: name -> (index in the state, arrivals per phase)
    names = ["dp_full", "s_loaded", "ds_free0", "ds_free1"] + [f"ds_full{i}" for i in range(n_ds)]
    need = {n: 1 for n in names}
    need["s_loaded"] = WARPS
    need.update({f"ds_full{i}": WARPS for i in range(n_ds)})
    index = {n: i for i, n in enumerate(names)}

    # A barrier is (phases completed modulo 4, arrivals of the current phase).
    def arrive(bars, name):
        phases, count = bars[index[name]]
        count += 1
        state = ((phases + 1) % 4, 0) if count == need[name] else (phases, count)
        return bars[: index[name]] + (state,) + bars[index[name] + 1:]

    def passed(bars, name, parity):  # mbarrier.try_wait.parity
        return bars[index[name]][0] % 2 != parity

    # warp: (block, step), step 0 wait dp_full + load + arrive s_loaded, 1 write packed dS, 2 arrive ds_full
    # ss:   (block, step), step 0 wait s_loaded(g-1), 1 wait ds_free(g-2), 2 issue + commit
    # acc:  (block, step), step 0 wait ds_full(g) and issue dQ(g)
    # pipes: number of products in flight per issuing thread
    # packed[u][w]: block whose dS warp w last wrote into buffer u
    start = (((0, 0),) * WARPS, (0, 0), 0, 0, 0, tuple((-1,) * WARPS for _ in range(2)), tuple((0, 0) for _ in names))
    seen, todo = {start}, [start]
    while todo:
        warps, ss, acc, ss_flying, dq_flying, packed, bars = todo.pop()
        nexts = []
        for w, (g, step) in enumerate(warps):
            if g == BLOCKS:
                continue
            new_packed, new_bars = packed, bars
            if step == 0:
                if not passed(bars, "dp_full", g % 2):
                    continue
                new_bars = arrive(bars, "s_loaded")
            elif step == 1:
                u = g % 2
                in_flight = [b for b in range(acc - dq_flying, acc) if b % 2 == u]
                if in_flight:
                    raise _Fault(f"dS({g}) written over dS({in_flight[0]}) in use")
                row = packed[u][:w] + (g,) + packed[u][w + 1:]
                new_packed = (row, packed[1]) if u == 0 else (packed[0], row)
            else:
                new_bars = arrive(bars, f"ds_full{g % n_ds}")
            moved = (g, step + 1) if step < 2 else (g + 1, 0)
            nexts.append((warps[:w] + (moved,) + warps[w + 1:], ss, acc, ss_flying, dq_flying, new_packed, new_bars))
        g, step = ss
        if g < BLOCKS:
            if step == 0 and (g == 0 or passed(bars, "s_loaded", (g - 1) % 2)):
                nexts.append((warps, (g, 1), acc, ss_flying, dq_flying, packed, bars))
            elif step == 1 and (g < 2 or passed(bars, f"ds_free{g % 2}", (g // 2 - 1) % 2)):
                nexts.append((warps, (g, 2), acc, ss_flying, dq_flying, packed, bars))
            elif step == 2:
                nexts.append((warps, (g + 1, 0), acc, ss_flying + 1, dq_flying, packed, bars))
        if acc < BLOCKS and passed(bars, f"ds_full{acc % n_ds}", (acc // n_ds) % 2):
            if packed[acc % 2] != (acc,) * WARPS:
                raise _Fault(f"dQ({acc}) issued on dS of blocks {packed[acc % 2]}")
            nexts.append((warps, ss, acc + 1, ss_flying, dq_flying + 1, packed, bars))
        if ss_flying:
            nexts.append((warps, ss, acc, ss_flying - 1, dq_flying, packed, arrive(bars, "dp_full")))
        if dq_flying:
            done = acc - dq_flying  # the oldest product in flight
            nexts.append((warps, ss, acc, ss_flying, dq_flying - 1, packed, arrive(bars, f"ds_free{done % 2}")))
        if not nexts and (acc < BLOCKS or any(b < BLOCKS for b, _ in warps)):
            raise _Fault(f"stuck: warps {warps}, dQ({acc}) next")
        for s in nexts:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return len(seen)


def _walk_v_tail(n_fixed):
    """Items of one block, the shortest way from one tail to the next.  The loads and the zeroing are the producer's step itself."""
    # barriers with one arrival a phase: the number of phases completed
    start = (0, 0, 0, (0,) * n_fixed, 0)  # producer item, issuing thread (2 * item + step), S products in flight, phases
    seen, todo = {start}, [start]
    while todo:
        item, issue, flying, fixed, q_empty = todo.pop()
        nexts = []
        # wait for q_empty of the item before, load Q, K and V, zero the tail, arrive
        if item < ITEMS and (item == 0 or q_empty % 2 != (item - 1) % 2) and item <= issue // 2 + 1:  # two items are published
            u = item % n_fixed
            nexts.append((item + 1, issue, flying, fixed[:u] + (fixed[u] + 1,) + fixed[u + 1:], q_empty))
        n, step = divmod(issue, 2)
        if n < ITEMS:
            if step == 0 and item > n:  # the tiles are there: issue S, commit q_empty
                nexts.append((item, issue + 1, flying + 1, fixed, q_empty))
            elif step == 1 and fixed[n % n_fixed] % 2 != (n // n_fixed) % 2:  # issue PV
                if fixed[n % n_fixed] <= n // n_fixed:
                    raise _Fault(f"PV of item {n} issued on a tail that is not zeroed")
                nexts.append((item, issue + 1, flying, fixed, q_empty))
        if flying:
            nexts.append((item, issue, flying - 1, fixed, q_empty + 1))
        if not nexts and n < ITEMS:
            raise _Fault(f"stuck: item {n} waits for its tail, the producer is at item {item}")
        for s in nexts:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return len(seen)


def _walk_deferred_store(lengths, gate, n_tail, slots):
    """dQ of an item is read by the elementwise warps at the end of the first block of the next item (or at the very end); every item
    has a tail to zero.  gate: the accumulating thread waits until it has been read; n_tail: barriers of the zeroed tail in turn;
    slots: items published at a time.  Faults: an accumulator written before it is read, a wait that never ends."""
    first = [sum(lengths[:k]) for k in range(len(lengths))]
    total, items = sum(lengths), len(lengths)
    item_of = [k for k, n in enumerate(lengths) for _ in range(n)]
    names = ["dp_full", "s_loaded", "ds_free0", "ds_free1", "ds_full0", "ds_full1", "acc_full", "acc_free"] + [f"tail{i}" for i in range(n_tail)]
    need = {n: WARPS if n in ("s_loaded", "ds_full0", "ds_full1", "acc_free") else 1 for n in names}
    index = {n: i for i, n in enumerate(names)}

    def arrive(bars, name):
        phases, count = bars[index[name]]
        state = ((phases + 1) % 4, 0) if count + 1 == need[name] else (phases, count + 1)
        return bars[: index[name]] + (state,) + bars[index[name] + 1:]

    def passed(bars, name, phase):
        return bars[index[name]][0] % 2 != phase % 2

    # warp: (block, step), steps 0 load, 1 dS handed over, 2 read dQ of the item before; block `total`: only step 2 is left
    start = (((0, 0),) * WARPS, 0, 0, 0, 0, 0, tuple((0, 0) for _ in names))
    seen, todo = {start}, [start]
    while todo:
        state = todo.pop()
        warps, prod, ss, acc, ss_flying, dq_flying, bars = state
        nexts = []
        read = lambda w: (item_of[w[0]] if w[0] < total else items) - (1 if w[1] < 3 else 0)  # noqa: E731  items a warp has read
        done = [read(w) if w[0] < total and w[0] == first[item_of[w[0]]] else item_of[w[0]] if w[0] < total else
                items - (w[1] < 3) for w in warps]
        for w, (g, step) in enumerate(warps):
            put = lambda v, b: nexts.append((warps[:w] + (v,) + warps[w + 1:], prod, ss, acc, ss_flying, dq_flying, b))  # noqa: E731
            starts = g < total and g == first[item_of[g]] and g > 0
            if g < total and step == 0 and passed(bars, "dp_full", g):
                put((g, 1), arrive(bars, "s_loaded"))
            elif g < total and step == 1:
                put((g, 2) if starts else (g + 1, 2 if g + 1 == total else 0), arrive(bars, f"ds_full{g % 2}"))
            elif step == 2 and passed(bars, "acc_full", (items if g == total else item_of[g]) - 1):
                put((g, 3) if g == total else (g + 1, 2 if g + 1 == total else 0), arrive(bars, "acc_free"))
        # the tiles of an item: its slot is free, Q and dO of the item before have been read, its statistics too
        if prod < items and (prod < slots or min(done) > prod - slots) and (
                prod == 0 or (ss >= first[prod - 1] + lengths[prod - 1] and all(w[0] > first[prod - 1] or w[1] > 0 and w[0] == first[prod - 1] for w in warps))):
            nexts.append((warps, prod + 1, ss, acc, ss_flying, dq_flying, arrive(bars, f"tail{prod % n_tail}")))
        if ss < total and prod > item_of[ss] and (ss == 0 or passed(bars, "s_loaded", ss - 1)) and (
                ss < 2 or passed(bars, f"ds_free{ss % 2}", ss // 2 - 1)):
            nexts.append((warps, prod, ss + 1, acc, ss_flying + 1, dq_flying, bars))
        if acc < total and passed(bars, f"ds_full{acc % 2}", acc // 2):
            k = item_of[acc]
            begins, ends = acc == first[k], acc == first[k] + lengths[k] - 1
            if (not ends or passed(bars, f"tail{k % n_tail}", k // n_tail)) and (
                    not (gate and begins and k > 0) or passed(bars, "acc_free", k - 1)):
                if begins and min(done) < k:
                    raise _Fault(f"dQ of item {k} written over that of item {min(done)}")
                nexts.append((warps, prod, ss, acc + 1, ss_flying, dq_flying + 1, bars))
        if ss_flying:
            nexts.append((warps, prod, ss, acc, ss_flying - 1, dq_flying, arrive(bars, "dp_full")))
        if dq_flying:
            g = acc - dq_flying
            after = arrive(bars, f"ds_free{g % 2}")
            if g == first[item_of[g]] + lengths[item_of[g]] - 1:
                after = arrive(after, "acc_full")
            nexts.append((warps, prod, ss, acc, ss_flying, dq_flying - 1, after))
        if not nexts and any(w != (total, 3) for w in warps):
            raise _Fault(f"stuck: warps {warps}, dQ({acc}) next, producer at item {prod}")
        for n in nexts:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return len(seen)


def _item_slots():
    return int(re.search(r"constexpr int kItemSlots = (\d+);", (CSRC / "bwd_sm100.cu").read_text()).group(1))


LENGTHS = [(1, 1, 1, 1, 1, 1, 1), (2, 1, 1, 2, 1, 1), (1, 3, 1, 1, 2)]


@pytest.mark.parametrize("lengths", LENGTHS)
def test_dq_of_an_item_is_stored_before_the_next_one_writes_over_it(lengths):
    assert re.search(r"&xb->acc_free, na & 1", (CSRC / "bwd_sm100.cu").read_text())
    assert _walk_deferred_store(lengths, True, _item_slots(), _item_slots()) > 20


def test_the_deferred_store_needs_its_barriers():
    with pytest.raises(_Fault, match="written over"):
        _walk_deferred_store(LENGTHS[0], False, 3, 3)
    with pytest.raises(_Fault, match="stuck"):
        _walk_deferred_store(LENGTHS[0], True, 1, 3)


PARTS = 3


def _walk_arrivals(own_counters, ordered=True):
    """Two calls on two streams, in each of which PARTS CTAs share a sequence (decode_balanced_kernel, csrc/kvcache_sm100.cu): a kernel
    that zeroes the counter, CTAs that store their part and count themselves, and the last of them merges.  own_counters: each call
    counts in its own scratch memory; else both in one counter, zero at first and put back to zero by the CTA that merges.  ordered: the
    CTAs count only behind the kernel that zeroes (each may start before it has finished).  Faults: a merge of parts that are not there,
    a call that nobody merges."""
    # call: (zeroed?, step of each CTA: 0 store, 1 count, 2 merge, 3 done); counters: None is what the memory held before
    start = (((not own_counters, (0,) * PARTS),) * 2, (None, None) if own_counters else (0, 0), (0, 0))
    seen, todo = {start}, [start]
    while todo:
        calls, counters, merged = todo.pop()
        nexts = []
        for c, (zeroed, ctas) in enumerate(calls):
            at = c if own_counters else 0

            def put(new_ctas, value, merges, new_zeroed=zeroed):
                nexts.append((calls[:c] + ((new_zeroed, new_ctas),) + calls[c + 1:], counters[:at] + (value,) + counters[at + 1:],
                              merged[:c] + (merged[c] + merges,) + merged[c + 1:]))

            if not zeroed:
                put(ctas, 0, 0, True)
            for i, step in enumerate(ctas):
                moved = lambda to: ctas[:i] + (to,) + ctas[i + 1:]  # noqa: E731
                if step == 0:
                    put(moved(1), counters[at], 0)
                elif step == 1 and (zeroed or not ordered):
                    old = counters[at]
                    put(moved(2 if old == PARTS - 1 else 3), None if old is None else old + 1, 0)
                elif step == 2:
                    if 0 in ctas:
                        raise _Fault(f"call {c} merges parts that are not there")
                    put(moved(3), counters[at] if own_counters else 0, 1)
        if not nexts and merged != (1, 1):
            raise _Fault(f"merges: {merged}")
        for n in nexts:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return len(seen)


def test_arrivals_are_counted_in_the_scratch_memory_of_the_call():
    source = (CSRC / "kvcache_sm100.cu").read_text()
    shared = re.search(r"arrivals = next_\w+\(\)", source) is not None
    wait = re.search(r"grid_dependency_wait\(\);[^\n]*\n\s*bars->last = atomic_add", source) is not None
    assert _walk_arrivals(not shared, shared or wait) > 100


def test_arrivals_need_counters_of_their_own_and_the_wait():
    with pytest.raises(_Fault, match="not there|merges:"):
        _walk_arrivals(False)
    with pytest.raises(_Fault, match="merges:"):
        _walk_arrivals(True, ordered=False)


def _walk_give_up(agree, warps=3, seqs=2, waits=2):
    """Consumer warps of decode_balanced_kernel (csrc/kvcache_sm100.cu) when bounded waits run out: per sequence `waits` of them, each
    of which a warp may give up or see complete, whatever the others see, then the barriers of the merge, which have no limit.  agree: every
    warp goes to the first of these, and all leave if one has given up; else a warp that gives up goes to the end of the kernel at once.
    Fault: a warp that waits at a barrier for one that does not come."""
    merge = 2  # barriers of a merge
    end = (seqs, 0, True)
    start = ((0, 0, True),) * warps  # sequence, step (waits, then barriers), no wait given up
    seen, todo = {start}, [start]
    while todo:
        state = todo.pop()
        nexts = []
        for w, (seq, step, ok) in enumerate(state):
            if seq < seqs and step < waits:
                gave_up = (seq, waits, False) if agree else end
                for to in ((seq, step + 1, ok), gave_up):
                    nexts.append(state[:w] + (to,) + state[w + 1:])
        at = [(seq, step) for seq, step, _ in state if seq < seqs]
        if len(at) == warps and len(set(at)) == 1 and at[0][1] >= waits:  # all are at the same barrier
            seq, step = at[0]
            if not all(ok for _, _, ok in state):
                nexts.append((end,) * warps)
            else:
                nexts.append(((seq, step + 1, True) if step + 1 < waits + merge else (seq + 1, 0, True),) * warps)
        if not nexts and any(w != end for w in state):
            raise _Fault(f"stuck: {state}")
        for n in nexts:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return len(seen)


def test_consumers_that_give_up_leave_together():
    body = re.search(r"decode_balanced_kernel\(const.*?\n\}\n", (CSRC / "kvcache_sm100.cu").read_text(), re.S).group(0)
    merge = body[body.index("WarpRows<D> mine"):]
    first = re.search(r"named_barrier_\w+\([^;]*;", merge)
    leaves = [m for m in re.finditer(r"\bbreak;", merge[:first.start()])]
    # the only way out ahead of the barrier is that of the tile loop
    agree = first.group(0).startswith("named_barrier_and") and len(leaves) == 1 and "ok = ok && wait_full(i);" in merge[:first.start()]
    assert _walk_give_up(agree) > 100


def test_a_consumer_that_leaves_by_itself_is_waited_for():
    with pytest.raises(_Fault, match="stuck"):
        _walk_give_up(False)


HANDOVERS = [(_walk_dq, "bwd_sm100.cu", "DqBarriers", "ds_full"), (_walk_v_tail, "fwd_sm100.cu", "Barriers", "v_fixed")]


@pytest.mark.parametrize("walk,source,struct,name", HANDOVERS)
def test_no_interleaving_breaks_the_hand_over(walk, source, struct, name):
    assert walk(_barriers(source, struct, name)) > 20


@pytest.mark.parametrize("walk,source,struct,name", HANDOVERS)
def test_one_barrier_would_not_do(walk, source, struct, name):
    with pytest.raises(_Fault):
        walk(1)
