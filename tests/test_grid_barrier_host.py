"""The grid barrier's memory ordering, read from its source: the arrival and the poll that sees it
have to be strong operations on the same bytes. Operations of different sizes that overlap in part
order nothing between blocks (PTX memory model, "morally strong operations"), so the width of the
release, the width of the acquire, and the accesses of the word they share are checked here, without
running it."""
import os
import re

from conftest import ROOT

CUDA = os.path.join(ROOT, "scout_b200", "csrc", "cuda")


def _code(name):
    text = open(os.path.join(CUDA, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def test_arrival_and_poll_have_one_width():
    code = _code("common.cuh")
    release = re.findall(r"atom\.add\.release\.gpu\.global\.(\w+)", code)
    acquire = re.findall(r"ld\.acquire\.gpu\.global\.(\w+)", code)
    assert release == acquire == ["u64"]
    body = code[code.index("bool grid_sync("):]
    body = body[:body.index("\n}\n")]
    assert len(re.findall(r"atom_add_release_gpu\(", body)) == 1 and len(re.findall(r"ld_acquire_gpu\w*\(", body)) == 1
    # both on the same address, and nothing else touches the word's halves during a launch
    assert re.findall(r"(?:atom_add_release_gpu|ld_acquire_gpu\w*)\((\w+)", body) == ["word", "word"]
    for name in sorted(os.listdir(CUDA)):
        if name.endswith((".cu", ".cuh")):
            assert not re.search(r"atomic\w+\(\s*&\w+->(count|err)\b\s*,\s*0, (1|code)", _code(name)), name
