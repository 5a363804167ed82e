"""Set-up of device memory in the library's source is done when it returns.

cudaMemset and cudaMemcpy from pageable memory run on the null stream and may
return before the device is done; the library's streams, a service's and a
batch's side streams and most callers' are not ordered after the null stream.
The words set up that way (scan counts and flags, descriptors, work lists)
are read by the next launch, so every such call goes through fill_now or
upload_now, which wait.
"""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hypergeometrica_gb300", "csrc")


def test_fills_and_uploads_wait():
    bare = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*h"))):
        text = "\n".join(line.split("//")[0] for line in open(path).read().splitlines())
        text = re.sub(r"inline cudaError_t (fill|upload)_now.*?\n}", "", text, flags=re.S)
        bare += [(os.path.basename(path), m) for m in re.findall(r"cudaMem(?:set|cpy)\([^;]*", text)]
    assert not bare, bare
