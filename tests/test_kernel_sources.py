"""Rules of the memory model that no run on today's hardware can show broken, checked in the
kernels' sources (no GPU needed)."""
import os
import re

import pytest

from conftest import PKG_DIR

CSRC = os.path.join(PKG_DIR, "csrc")
KERNELS = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def body(text, start):
    """The braces that follow `start`."""
    i = text.index("{", text.index(start))
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise AssertionError("unbalanced braces after " + start)


@pytest.mark.parametrize("name", KERNELS)
def test_no_writer_is_elected_among_whoever_arrives(name):
    """__activemask() need not name all lanes of a branch: two parties of one branch would each elect
    a writer for the same entry of a shared table."""
    assert not re.search(r"__(match_any|match_all|shfl\w*|reduce\w*)_sync\s*\(\s*__activemask", source(name))


def test_the_normal_tables_writes_are_ordered_before_the_next_reads():
    """A vote orders no memory: between an entry's two writes and the next brick's reads of the table
    stands a __syncwarp, and one stands between a brick's reads and the writes after them."""
    kernel = body(source("vx_payload.cu"), "build_normals_kernel(")
    loop = body(kernel, "for (uint32_t brick")
    read, kept, queue = loop.rindex("w.block[at]"), loop.index("keep("), loop.rindex("w.queue_at[")
    assert "__syncwarp()" in loop[read:kept]
    assert "__syncwarp()" in loop[queue:loop.index("drain(", queue)]
    assert queue > kept
    drain = body(kernel, "auto drain")
    assert "__syncwarp()" in drain[drain.index("keep("):]


WIDTH = {"unsigned char": 1, "uint8_t": 1, "uint16_t": 2, "uint32_t": 4, "float": 4, "float2": 8, "uint2": 8,
         "unsigned long long": 8, "uint64_t": 8, "float4": 16, "uint4": 16}


@pytest.mark.parametrize("name", KERNELS)
def test_shared_arrays_read_by_wider_words_say_their_alignment(name):
    """A static shared array is aligned to its elements and no more, wherever the compiler happens to
    place it: one that is accessed through a pointer to a wider type has to ask for the alignment."""
    text = source(name)
    for to, array in re.findall(r"reinterpret_cast<\s*(?:const\s+)?([\w ]+?)\s*\*>\s*\(\s*&?(\w+)", text):
        for align, of in re.findall(r"(?<!extern )__shared__\s+(?:__align__\((\d+)\)\s+)?([\w ]+?)\s+%s\s*\[" % array, text):
            if to in WIDTH and of in WIDTH and WIDTH[to] > WIDTH[of]:
                assert align and int(align) >= WIDTH[to], f"{name}: {array}"
