"""The kernels after the narrowphase trust a pair's contact count to be at
most four (they index four rows and points a pair with it), so a generator's
negative count must never be stored.  Every store of a count is in
store_contacts, which turns it into the step's error."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fyzzxyzzy-sdk_b200", "csrc")


def test_counts_are_stored_through_the_check():
    stores = []
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        function = ""
        for line in open(path):
            m = re.match(r"(?:template .*)?(?:__device__|__global__|static|void|inline).*?(\w+)\(", line)
            function = m.group(1) if m else function
            if re.search(r"\bcur\.count\[[^]]*\]\s*=[^=]", line):
                stores.append((os.path.basename(path), function))
    assert stores == [("narrowphase.cu", "store_contacts")]
    source = open(os.path.join(CSRC, "narrowphase.cu")).read()
    body = source[source.index("void store_contacts("):]
    body = body[:body.index("\n}\n")]
    check = re.search(r"if \(count < 0\) \{\s*atomicOr\(s\.err, kErrContactOverflow\);\s*count = 0;\s*\}", body)
    assert check and check.end() < body.index("cur.count[")
