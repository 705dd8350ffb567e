"""What no run may show, since a violation could hang or fault the GPU, read from the kernels' sources."""
import glob
import os
import re

import pytest

from nanoserve_b200 import build

SOURCES = {os.path.basename(f): open(f).read() for f in sorted(glob.glob(os.path.join(build.CSRC, "*.cu")))}


@pytest.mark.parametrize("name", [n for n, s in SOURCES.items() if "poisoned" in s])
def test_named_barriers_and_the_status_word(name):
    """Another CTA may set the status word at any time and a named barrier is unbounded.  Either one thread reads the word ahead
    of a __syncthreads and the whole CTA decides by that value, or every warp reads it for itself and meets each named barrier
    of the skipped work all the same."""
    body = SOURCES[name]
    read = re.search(r"\*reinterpret_cast<volatile int\*>\(p\.status\)", body)
    decision = body.index("const bool poisoned = ")
    assert len(re.findall(r"\*\>\(p\.status\)", body)) == 1
    if read.start() < decision:
        assert re.search(r"if \(tid == \d+\) \*status_seen = $", body[:read.start()])
        assert "__syncthreads();" in body[read.start():decision]
        assert body.startswith("const bool poisoned = *status_seen != 0;", decision)
    else:
        assert body.startswith("const bool poisoned = __any_sync(", decision)
        work, skipped = body[decision:].split("\n  } else if (p.ks == 1 && warp < kMain) {", 1)
        skipped = skipped[:skipped.index("\n  }\n")]
        assert "\n  if (!poisoned) {\n" in work and "bar.sync" not in body[decision + len(work) + len(skipped) + 60:]
        barriers = [re.findall(r'asm volatile\("(bar\.sync[^;]*);', part) for part in (work, skipped)]
        assert len(barriers[0]) == 1 == len(barriers[1])


def test_scale_prefetches_are_bounded():
    """A step index taken from the CTA's share of K may lie one pair of steps behind a weight row's scales (a share of one pair
    has nothing for the second group of warps): behind the last row that is past the end of S."""
    K = 256  # one pair of steps; the second group's first step
    assert 2 * (0 + 1) >= K // 128
    guards = [re.findall(r"if \(([^{}]*?)\) prefetch_l2\(s_row \+ (\w+)\)", s) for s in SOURCES.values()]
    found = [(cond, at) for g in guards for cond, at in g]
    assert len(found) == sum(s.count("prefetch_l2(s_row") for s in SOURCES.values()) >= 2
    for cond, at in found:
        assert re.search(r"\b%s < p\.KG" % at, cond), (cond, at)


def test_scale_prefetches_by_other_warps_are_bounded():
    """The warps that issue the products prefetch the sector ahead of step i for rows of their tile: a row and a step that exist."""
    found = [m for s in SOURCES.values() for m in re.finditer(r"prefetch_l2\(p\.S \+ \(size_t\)n \* p\.KG \+ ([^;]*)\);", s)]
    assert len(found) == sum(s.count("prefetch_l2(p.S") for s in SOURCES.values()) == 2
    for m in found:
        before = m.string[:m.start()]
        assert before.endswith("if (n < p.N) ")
        step = re.findall(r"if \(([^{}]*)\) \{", before)[-1]
        assert step in ("(i & 7) == 0 && i + 8 < np", "i % kSectorSteps == 0 && i + kSectorSteps < nkb")
        assert m.group(1) == ("2 * (pr0 + i) + 16" if "np" in step else "(kb0 + i + kSectorSteps) * (128 / MODE)")


def test_questions_ahead_of_work_do_not_wait():
    """A try_wait may suspend the warp for a while: an answer that is only used behind a block's conversion is asked for by
    test_wait, and try_wait stands where nothing else is left to do (in the waits of ptx.cuh and in pairs of questions)."""
    for name, s in SOURCES.items():
        assert not re.search(r"= mbar_try_wait\(", s), name
