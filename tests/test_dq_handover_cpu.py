"""The hand-over of dS in the dQ kernel (bwd_dq_kernel, csrc/bwd_sm100.cu), walked through exhaustively.

The model has the kernel's waits and arrivals for one long item: two elementwise warps, the thread that issues S and dP, the one
that issues dQ, and the tensor pipe, which completes each thread's products in order and as late as it likes.  Barriers behave as
mbarriers do: a phase ends with the last expected arrival, and a wait sees only the parity of the phase.  Every interleaving is
visited.  The number of ds_full barriers is read from the kernel's source.
"""
import re
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parents[1] / "flash_attention_turing_b200" / "csrc" / "bwd_sm100.cu"
WARPS = 2
BLOCKS = 6


def _ds_full_barriers():
    text = SOURCE.read_text()
    fields = re.search(r"struct DqBarriers \{(.*?)\n\};", text, re.S).group(1)
    own = re.search(r"\bds_full\[(\d+)\]", fields)
    return int(own.group(1)) if own else 1


class _Fault(Exception):
    pass


def _walk(n_ds):
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


def test_no_interleaving_breaks_the_hand_over():
    assert _walk(_ds_full_barriers()) > 100


def test_one_barrier_for_all_blocks_would_not_do():
    with pytest.raises(_Fault):
        _walk(1)
