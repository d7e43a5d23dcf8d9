"""The MMA issuer looks at several barriers at once, a lane each, and one elected lane issues.
A warp vote carries the answers but orders no memory, so between the vote and the first MMA
there has to be a ``__syncwarp`` (which does): without it the issuing lane never acquired the
barriers that other lanes saw - the next K tile, O read out - and its MMAs race with the writes
behind them.  Nothing on a GPU shows such a race reliably; the order is read off the source
(megaattention_b200/csrc/fused_prefill.cu)."""
import os
import re

SRC = os.path.join(os.path.dirname(__file__), "..", "megaattention_b200", "csrc", "fused_prefill.cu")


def _code():
    text = open(SRC).read()
    return re.sub(r"//[^\n]*", "", text)


def test_votes_over_barriers_are_followed_by_a_warp_barrier():
    code = _code()
    votes = [m.end() for m in re.finditer(r"__(?:all|any)_sync\(0xffffffffu, mbar_test_wait\(", code)]
    assert votes, "the combined look at the operands' barriers is not where this test expects it"
    for at in votes:
        first_mma = re.compile(r"issue_(?:pv|qk)|mma_(?:ss|ts)\(").search(code, at).start()
        between = code[at:first_mma]
        assert "__syncwarp();" in between
        # at the level of the vote's own statement: not inside the branch of a failed vote
        depth, found = 0, False
        for tok in re.finditer(r"[{}]|__syncwarp\(\);", between):
            if tok.group() == "{":
                depth += 1
            elif tok.group() == "}":
                depth -= 1
            elif depth == 0:
                found = True
        assert found
