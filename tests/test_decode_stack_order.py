"""Order of the whole-stack decode kernel's accesses to memory that its warps share, read from its source: what it would take to
see one of these faults on a device is a matter of timing."""
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parent.parent / "sensenova_u1_b200" / "csrc" / "decode_stack.cu").read_text()


def _body(name):
    """Code of the function ``name``, without comments, from its opening to its closing brace."""
    code = re.sub(r"//[^\n]*", "", SOURCE)
    at = code.index("{", re.search(rf"\b{name}\(const Args& a[^;{{]*\)\s*{{", code).start())
    depth = 0
    for i in range(at, len(code)):
        depth += {"{": 1, "}": -1}.get(code[i], 0)
        if depth == 0:
            return code[at:i + 1]
    raise AssertionError(name)


def _constant(name):
    return int(re.search(rf"constexpr int {name} = (\d+)", SOURCE).group(1))


@pytest.mark.parametrize("rows,reduction", [(2, 1024), (1, 2048), (1, 4096), (2, 4096)])
def test_attention_is_through_with_its_sums_before_the_next_product_stores_x(rows, reduction):
    warps, chunk, heads = _constant("CW"), _constant("KC"), _constant("HG")
    # bytes of ``red`` that a warp reads (two results per thread out of every warp's 128 per head) and of its rows of x
    reads = [{w * heads * 512 + (warp * 64 + i) * 4 for w in range(warps) for i in range(64)} for warp in range(warps)]
    part = reduction // chunk * rows * (chunk // warps * 2)
    stores = [range(warp * part, (warp + 1) * part) for warp in range(warps)]
    shared = any(b in stores[w] for w in range(warps) for o in range(warps) if o != w for b in reads[o])
    assert shared                                   # the two do lie over one another: only a barrier keeps them apart
    body = _body("attend")
    after = body[body.rindex("red +"):]
    depth, least = 0, 0
    for m in re.finditer(r"[{}]|named_bar_sync\(1, CT\);", after):
        depth += {"{": 1, "}": -1}.get(m.group(), 0)
        least = min(least, depth)
        if m.group().startswith("named") and depth == least:
            break                                   # in no branch that was opened after the read
    else:
        pytest.fail("no barrier of all consumer warps between the sums and the end of the attention")


def test_a_word_between_ctas_is_one_element_of_64_bits():
    code = re.sub(r"//[^\n]*", "", SOURCE)
    accesses = re.findall(r"(?:ld|st)\.(?:relaxed|volatile|acquire|release)\.gpu\.[\w.]+", code)
    assert sorted(accesses) == ["ld.relaxed.gpu.global.b64", "ld.relaxed.gpu.global.v2.b64", "st.relaxed.gpu.global.b64"]
    for name in ("x", "x1", "qkv", "o", "act", "part"):             # and nothing else touches the words
        assert not re.search(rf"\*\s*\(?(?:reinterpret_cast<[^>]*>\()?a\.{name}\b", code)
