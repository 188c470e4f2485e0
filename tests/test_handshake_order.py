"""What the ranges of a run read of one another, against what their publication
releases (no GPU): the kernel source's stores, fence and loads in order.

A reader of the count of published ranges may see the increment before any store
that no fence separates from it, so everything it reads must be stored before the
publication's last fence; the tagged word lies behind that fence and is only for a
reader that acquires that very word."""
import pathlib
import re

import pytest

SRC = pathlib.Path(__file__).resolve().parent.parent / "apsep_gb300" / "csrc" / "apsep_range_kernel.cuh"


def _code() -> str:
    text = SRC.read_text()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def _block(code: str, head: str) -> str:
    """The braced block that follows the first match of `head`."""
    at = re.search(head, code)
    assert at, head
    start = code.index("{", at.end() - 1)
    depth = 0
    for i in range(start, len(code)):
        depth += {"{": 1, "}": -1}.get(code[i], 0)
        if depth == 0:
            return code[start:i + 1]
    raise AssertionError("unbalanced: " + head)


def _publication():
    """Words stored before the fence, and behind it, by range_publish."""
    body = _block(_code(), r"void range_publish\(")
    count = body.index("red_add_u32(&a.s.ctr->finished")
    fences = [m.start() for m in re.finditer(r"fence_acq_rel\(\)|__threadfence\(\)", body[:count])]
    assert fences, "no fence before the count"
    words = r"a\.s\.(range_state|range_key|group_min)\b"
    return set(re.findall(words, body[:fences[-1]])), set(re.findall(words, body[fences[-1]:count]))


READERS = {
    "range_min": r"T range_min\(",
    "group_min_of": r"T group_min_of\(",
    "answer_before": r"int answer_before\(",
    "from_ready": r"auto from_ready = \[&\]\(\) \{",
}


@pytest.mark.parametrize("reader", sorted(READERS))
def test_readers_of_the_count_read_released_words(reader):
    released, behind = _publication()
    body = _block(_code(), READERS[reader])
    body += "".join(_block(_code(), READERS[f]) for f in ("range_min", "group_min_of")
                    if f != reader and re.search(r"\b%s<" % f, body))
    read = set(re.findall(r"a\.s\.(range_state|range_key|group_min)\b", body))
    assert not read & behind, "%s reads %s, which no fence orders before the count" % (reader, read & behind)
    assert read <= released | {"group_min"}


def test_lanes_are_ordered_before_they_read_what_others_acquired():
    body = _block(_code(), r"void range_prefix\(")
    won = _block(body[body.index("range_state"):], r"if \(__all_sync\(FULL, ok\)\) \{")
    assert "__syncwarp()" in won[:won.index("range_min<")]


def test_tagged_words_are_acquired():
    code = _code()
    loads = [m.start() for m in re.finditer(r"a\.s\.range_state\b", code)]
    publish = _block(code, r"void range_publish\(")
    at = code.index(publish)
    for i in loads:
        line = code[code.rfind("\n", 0, i) + 1:code.find("\n", i)]
        stored = at <= i < at + len(publish) or re.search(r"range_state\[i\] = 0", line)
        assert stored or "ld_acquire_u64" in line, line.strip()
