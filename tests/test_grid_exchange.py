"""The exchange entries of the resident grid form are their own flags: a reader takes an entry
as soon as it differs from the unset value.  That holds only if an entry is seen whole or not at
all.  The memory model makes a vector access one access per element, so every access to an
exchange word must have elements as wide as the entries: b32 for FP32, b64 for FP64.  A torn
entry cannot be provoked, so the accesses themselves are checked."""
import os
import re

from conftest import PKG


def source():
    with open(os.path.join(PKG, "csrc", "dmm_grid.cuh")) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_vector_accesses_have_whole_entries_as_elements():
    text = source()
    found = re.findall(r"\b(ld|st)\.relaxed\.gpu\.global\.(v\d)\.([a-z]\d+)", text)
    assert sorted(found) == [("ld", "v2", "b64"), ("ld", "v4", "b32"),
                             ("st", "v2", "b64"), ("st", "v4", "b32")]
    # each in the branch of its precision: FP32 first
    for op in ("ld", "st"):
        body = text[text.index(f" {op}_word("):]
        body = body[:body.index("\n}\n")]
        assert "sizeof(T) == 4" in body
        assert body.index(f"{op}.relaxed.gpu.global.v4.b32") < body.index("else") < body.index(
            f"{op}.relaxed.gpu.global.v2.b64")


def test_every_access_names_the_type_of_its_entries():
    text = source()
    uses = re.findall(r"\b(?:ld_word|st_word|word_set|unset_word|take_words)\b(<[^>]*>)?\(", text)
    calls = [u for u in uses if u]
    assert len(calls) >= 8 and set(calls) == {"<T>"}
    # without a type: the five definitions only
    assert len([u for u in uses if not u]) == 5
