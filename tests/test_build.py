"""The two ways to build the libraries list the same files."""

import pytest

from megakernels_b200.build import CSRC, LIBRARIES


@pytest.mark.parametrize("name,sources,headers", [("llama", "SRC", "HDR"), ("hybrid", "HYBRID_SRC", "HYBRID_HDR")])
def test_makefile_lists_the_files_of_the_build(name, sources, headers):
    lists = {}
    for line in (CSRC / "Makefile").read_text().splitlines():
        if ":=" in line:
            key, value = line.split(":=", 1)
            lists[key.strip()] = set(value.split())
    assert lists[sources] == set(LIBRARIES[name].sources)
    assert lists[headers] == set(LIBRARIES[name].headers)
    assert all((CSRC / f).exists() for f in lists[sources] | lists[headers])
