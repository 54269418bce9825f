"""A role of a kernel whose bounded wait gave up issues nothing more: no later wait of the role may set its flag back.

In the sources an assignment `ok = warp_all(<wait>)` therefore stands under a condition that asks for `ok`, or where the last
thing said about `ok` was a loop condition, a `break` out or its declaration.  Read from the text, without a GPU: to make a
load fail to land on a device would be a fault."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "megakernel-exploration_b200", "csrc")
ASSIGN = re.compile(r"\bok = warp_all\(")
SAFE = re.compile(r"if \(!ok\b|^(for|while) \(.*\bok\b|\bbool ok\b")
LAMBDA = re.compile(r"\bauto \w+ = \[&\]")


def unguarded(text):
    """Line numbers of assignments that an earlier failed wait of the role does not keep from running.  (A lambda's first
    one is its callers'.)"""
    lines = [re.sub(r"//.*", "", line).strip() for line in text.splitlines()]

    def before(n):
        """The line above n that last spoke of `ok` or opened a lambda; branches that exclude n's are passed over."""
        depth, m = 0, n - 1
        if lines[n].startswith("else") or re.fullmatch(r"else\b.*", lines[m]):
            while not ASSIGN.search(lines[m]):
                m -= 1
            m -= 1
        while m >= 0:
            line = lines[m]
            if depth == 0 and line.startswith("} else"):
                inner = 1
                while inner:
                    m -= 1
                    inner += lines[m].count("}") - lines[m].count("{")
                continue
            if re.search(r"\bok\b", line) or (depth == 0 and LAMBDA.search(line)):
                return line
            depth = max(0, depth + line.count("}") - line.count("{"))
            m -= 1
        return ""

    bad = []
    for n, line in enumerate(lines):
        at = ASSIGN.search(line)
        if at and not re.search(r"\bok\b", line[:at.start()].replace("bool ok", "")):
            last = before(n)
            if not (SAFE.search(last) or LAMBDA.search(last)):
                bad.append(n + 1)
    return bad


def test_the_reading_finds_a_forgotten_wait():
    loop = "for (int i = 0; i < n && ok; ++i) {\n ok = warp_all(mbar_wait(a));\n for (int t = 0; t < 2; ++t) {\n %s ok = warp_all(mbar_wait(b));\n if (!ok) break;\n}\n}"
    assert unguarded(loop % "if (t == 0)") == [4]
    assert unguarded(loop % "if (ok && t == 0)") == []


@pytest.mark.parametrize("name", sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu*"))))
def test_no_wait_forgets_an_earlier_one(name):
    with open(os.path.join(CSRC, name)) as f:
        assert unguarded(f.read()) == []
