"""tcgen05.ld is a warp's instruction: all 32 lanes execute it together. Read off the source: where lanes may have parted
since the last one (pixels outside the image skip the epilogue), they meet again before the next."""
import os
import re

from test_cluster_barriers import CSRC, _body, _code

CONVERGES = r"__syncwarp\(|__all_sync\("


def test_lanes_meet_before_every_accumulator_read():
    assert os.path.isdir(CSRC)
    text = _code("lsb_unet.cu")
    for kernel in ("conv3x3_tc_kernel", "conv_dw_kernel"):
        body = _body(text, kernel)
        reads = [m.start() for m in re.finditer(r"tcgen05\.ld\.sync", body)]
        assert reads
        for at in reads:
            # back to the start of the innermost loop around it (or the lambda that holds it)
            depth, i = 0, at
            while depth < 1:
                i -= 1
                depth += (body[i] == "{") - (body[i] == "}")
                if depth == 1 and not re.search(r"(for \([^{}]*\)|\]\s*\([^{}]*\))\s*$", body[:i]):
                    depth = 0  # an if's or a plain block's brace: lanes do not part at a loop's end there
            loop = body[i:at]
            diverges = re.search(r"\bif \(!in\) continue", body[i:])
            assert not diverges or re.search(CONVERGES, loop), kernel
