"""Hand-over between the MMA lane and the softmax warps of one query tile in the tcgen05 prefill kernel, as a state machine of which every
interleaving is visited.  What it checks is the one thing that a wait by parity cannot see: that a barrier completes no second phase before every
warp has seen the first.  The number of barriers that the batches use in turn is read from the kernel's source."""
import os
import re

SOURCE = os.path.join(os.path.dirname(__file__), "..", "flash_attn_v100_b200", "csrc", "prefill_tc5_kernel.cuh")


def _stuck(bars, items=3, steps=2, warps=2):
    """A state from which nothing can go on although work is left, or None.

    Per item the MMA lane commits one batch with the first QK (it needs the Q buffer, which the softmax gives back when it sees the batch of the
    previous item's last QK) and one per step (it needs P of the step from every warp); a warp waits for the batch of a step, hands P over, and waits
    for the item's last batch before it goes on to the next item.  Batch c completes a phase of barrier c % bars; the wait for it passes
    unless the barrier's current phase has the parity of phase c // bars."""
    per = steps + 1                                        # batches per item, and waits of a warp per item
    start = (0,) * (1 + warps)                             # batches committed; waits that each warp is through with
    seen, todo = {start}, [start]
    while todo:
        state = todo.pop()
        done, through = state[0], state[1:]
        nexts = []
        if done < items * per:
            item, i = divmod(done, per)
            if i == 0:
                ready = item == 0 or through[0] >= item * per - 1          # the last step's wait of the previous item
            else:
                ready = all(w >= item * per + i for w in through)          # P of step i - 1 follows the wait for batch i - 1
            if ready:
                nexts.append((done + 1,) + through)
        for k, w in enumerate(through):
            if w < items * per:
                completed = (done - w % bars + bars - 1) // bars           # phases that barrier w % bars has behind it
                if (completed & 1) != ((w // bars) & 1):
                    nexts.append((done,) + through[:k] + (w + 1,) + through[k + 1:])
        if not nexts and state != (items * per,) * (1 + warps):
            return state
        for n in nexts:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return None


def test_one_barrier_is_not_enough():
    assert _stuck(1) is not None


def test_batch_barriers_of_the_kernel():
    bars = int(re.search(r"constexpr int kBatchBars = (\d+);", open(SOURCE).read()).group(1))
    for steps in (1, 2, 3):
        assert _stuck(bars, steps=steps) is None
