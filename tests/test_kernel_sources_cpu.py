"""What a kernel does before its dependency wait, read from its source: a race there shows on no CPU and rarely on a GPU."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "trapetum_b200" / "csrc"
# arrays of a call that the launch just before it in the stream may have written
CALL_ARRAYS = ("token_seq", "seq_start", "slot_ids", "len_after", "page_table", "state", "proj", "dt", "xbc", "y", "q", "k", "v",
               "pool", "partial", "chunk_state", "chunk_decay", "decay", "logits")


def kernels(source):
    """(name, text between the kernel's opening brace and its first pdl_wait()) of every kernel that waits."""
    for m in re.finditer(r"^(?:template[^\n]*\n)?__global__\s+void\s+(?:__launch_bounds__\([^\n]*?\)\s+)?(\w+)\([^{;]*\)\s*\{", source, re.M):
        body = source[m.end():]
        body = body[:body.index("\n}\n")]
        if "pdl_wait()" in body:
            yield m.group(1), body[:body.index("pdl_wait()")]


@pytest.mark.parametrize("name", ["mamba2", "gla", "attention_latent", "attention_mixed"])
def test_a_call_s_arrays_are_read_after_the_wait(name):
    """The first launch of a public call starts while the launch before it, which may build these arrays on the device, drains."""
    found = list(kernels((CSRC / f"{name}.cu").read_text()))
    assert found
    early = [(kernel, field) for kernel, text in found for field in CALL_ARRAYS
             if re.search(rf"\ba\.{field}\s*\[", re.sub(r"//[^\n]*", "", text))]
    assert early == []
