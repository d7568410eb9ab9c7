"""Which arrays the kernels read with __ldg (ld.global.nc): memory must be
read-only as long as a kernel that reads it so runs.  A violation need not show
in results, so the sources are looked at."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "recon_gb300", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def body(text, head):
    """The function that begins with `head`, up to the brace that closes it."""
    start = text.index(head)
    depth, k = 0, text.index("{", start)
    while True:
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        k += 1
        if depth == 0:
            return text[start:k]


def test_preparation_kernel_reads_what_it_wrote_with_plain_loads():
    code = body(source("kernels.cu"), "void student_body(")
    written = set(re.findall(r"\bd\.(icp_\w+)\[[^\]]*\]\s*=[^=]", code))
    assert {"icp_r2", "icp_mask", "icp_w"} <= written
    for name in written:
        assert not re.search(r"__ldg\([^;]*\bd\." + name, code), name


def test_schedule_reads_what_its_launches_write_past_the_read_only_path():
    """The launches of a frame overlap: a kernel is running while the one before
    it still writes."""
    text = source("kernels.cu")
    for head in ("k_icp_mask(const InstDesc *D", "k_icp_student_pass(const InstDesc *D", "void icp_chunks(",
                 "bool photo_cluster(", "void finalize_iter(", "void student_body("):
        code = body(text, head)
        pointers = "|".join(re.findall(r"\*(\w+)\s*=\s*d\.(?:icp_\w+|ph_\w+|fx)\b", code) + re.findall(
            r",\s*\*(\w+)\s*=\s*d\.icp_\w+", code)) or "none"
        for load in re.findall(r"__ldg\(([^;]*);", code):
            assert not re.search(r"\bd\.(icp_|ph_|fx\b|T\b|stats\b)|\b(" + pointers + r")\b", load), (head, load)


def test_listed_update_reads_its_list_with_plain_loads():
    """k_pick_blocks and k_update_list wait for the launch that writes what they
    read: no pointer to it promises (const and __restrict__) that it stays as it is."""
    text = source("tsdf.cu")
    assert not re.search(r"__ldg\([^;]*\b(far_tiles|list|counts?)\b", text)
    for head in ("k_pick_blocks(", "k_update_list(", "bool hidden("):
        params = re.search(re.escape(head) + r"([^)]*)\)", text).group(1)
        assert not re.search(r"__restrict__\s+(far_tiles|list|counts?)\b", params), head
