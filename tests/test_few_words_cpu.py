"""The order in which blocks of the few-sequence decode kernel use one another's words again, worked out on the CPU.

Words announce themselves, so what a block does with one has to be ordered against the same word's other uses by something
else: a block returns words to EMPTY two layers ahead, and every word serves again after RING layers.  The only order between
blocks that the memory model grants there is the counter: a fence of every block in the middle of a layer (`count`), and a
look at it in the middle of a later one (`settled`).  Here every event of a block stands in its program order, and an event
of one block counts as before an event of another only through such a fence and such a look.
"""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "async-gpu_b200", "csrc", "decode_few.cu")


def _source():
    with open(SOURCE) as f:
        return f.read()


def _events(layers, steps):
    """A block's events in order: (what, word, layer of the launch)."""
    ev = []
    for i in range(layers * steps):
        step, last = i // layers, i % layers == layers - 1
        if i % layers:
            ev.append(("read", "fp", i - 1))
        ev += [("publish", "qkv", i), ("reset", "qkv", i + 2), ("write", "row", i), ("reset", "att", i + 2)]
        ev += [("read", "row", j) for j in range(i % layers, i, layers)]
        ev += [("read", "qkv", i), ("publish", "att", i), ("look", "", i), ("read", "att", i), ("publish", "out", i),
               ("reset", "out", i + 2)]
        ev += [("read", "out", i), ("fence", "", i), ("publish", "fc", i), ("reset", "fc", i + 2)]
        ev += [("read", "fc", i), ("publish", "fp", i), ("reset", "fp", i + 2)]
        if last:
            ev += [("look", "", i + 1), ("read", "fp", i), ("publish", "pick", step), ("read", "pick", step), ("reset", "pick", step + 1)]
    return ev


@pytest.mark.parametrize("layers", [1, 2, 3, 5, 12])
def test_every_use_of_a_word_is_ordered_before_the_next(layers):
    s = _source()
    ring = int(re.search(r"constexpr int RING = (\d+)", s).group(1))
    assert "(rp + 2) % RING" in s  # words are returned two layers ahead
    assert "settled(wait, P.fenced, g == OUT ? all_fenced : all_fenced + nblk)" in s  # the looks' targets
    ev = _events(layers, 6)
    at = {e: n for n, e in enumerate(ev)}
    fences = [(n, i) for n, (what, _, i) in enumerate(ev) if what == "fence"]
    looks = [(n, i) for n, (what, _, i) in enumerate(ev) if what == "look"]

    def ordered(a, b):
        """Event a of one block before event b of another."""
        first = min((i for n, i in fences if n >= at[a]), default=None)
        seen = max((i for n, i in looks if n <= at[b]), default=0)  # a look waits for the fences of the layers before its own
        return first is not None and first < seen

    checked = 0
    for what, word, i in ev:
        if what == "reset" and ("read", word, i) in at:
            assert ordered((what, word, i), ("read", word, i)), f"{word} of layer {i}: an older value could be read"
            checked += 1
        if what == "reset":
            before = i - (2 if word == "pick" else ring)
            if ("read", word, before) in at:
                assert ordered(("read", word, before), (what, word, i)), f"{word} of layer {before}: taken back before it is read"
                checked += 1
    for i in range(layers * 6):
        for j in range(i + layers, layers * 6, layers):
            write, read = at[("write", "row", i)], [n for n, e in enumerate(ev) if e == ("read", "row", i)]
            assert all(min((k for n, k in fences if n >= write)) < max((k for n, k in looks if n <= r), default=0) for r in read)
            checked += 1
    assert checked > 20
