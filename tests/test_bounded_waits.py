"""Blocks that wind down when a wait runs out: read from the source, since no GPU is made to wait for nothing."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kvcache_b200", "csrc")


def _block(text, at):
    """The text between the brace at `at` and the one that closes it."""
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if not depth:
            return text[at + 1:i]
    raise AssertionError("no closing brace")


def _without_comments(text):
    return re.sub(r"//[^\n]*", "", text)


def test_softmax_warps_leave_the_line_of_work_together():
    """A tile's four softmax warps meet at named barriers, which have no limit.  A warp whose wait has run out may therefore leave the loop
    over the block's pieces only where all four do: after the barrier at which they tell one another."""
    with open(os.path.join(CSRC, "attention_pairs.cu")) as fh:
        text = _without_comments(fh.read())
    softmax = text[text.index("setmaxnreg.inc"):]
    pieces = _block(softmax, softmax.index("{", softmax.index("for (int w = w_begin; w < w_end && ok;)")))
    tiles_at = pieces.index("{", pieces.index("for (int i = 0; i < hf.n"))
    tiles = _block(pieces, tiles_at)
    assert "bar." not in tiles and "all_of_tile" not in tiles          # within the loop over key tiles: waits with a limit, and none on a barrier
    rest = pieces[tiles_at + len(tiles) + 2:]
    assert "bar.sync" in rest
    leave = [m.start() for m in re.finditer(r"\bbreak;", rest)]
    agreed = re.search(r"ok = all_of_tile\(1 \+ wg, ok\);\s*if \(!ok\) (break;)", rest)
    assert agreed and leave == [agreed.start(1)]
    assert rest.index("bar.sync") > agreed.start() and "ok =" not in rest[agreed.end():]


def test_copies_still_on_their_way_are_waited_for():
    """A block that gives up asks for nothing more and waits, with a limit, for the copies that it has asked for: shared memory that a copy
    still writes to must not go to the next block."""
    with open(os.path.join(CSRC, "latent_flash.cu")) as fh:
        text = _without_comments(fh.read())
    kernel = text[text.index("latent_rows16_kernel("):]
    tiles = _block(kernel, kernel.index("{", kernel.index("for (int tile = 0; tile < ntiles; ++tile)")))
    given_up = tiles.index("if (__syncthreads_or(!ok))")
    assert given_up < tiles.index("fetch(")                            # decided by all threads, before the next copies are asked for
    down = _block(tiles, tiles.index("{", given_up))
    assert "for (int c = tile; c < ntiles && c < max(LEAD, tile + STAGES - 1); ++c) tc::mbar_wait(" in down and "break;" in down

    with open(os.path.join(CSRC, "attention_pairs.cu")) as fh:
        text = _without_comments(fh.read())
    down = _block(text, text.index("{", text.index("if (sh.failed && tid == 0)")))
    for name in ("q_copies", "k_copies", "v_copies"):                  # the last copies by their own number, not a barrier's first phase
        assert name in down
    assert "full[h], 0)" not in down and "full[s], 0)" not in down
