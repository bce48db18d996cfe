"""The tridiagonalisation's values that carry their step's tag: a 64-bit element of an access is read
and written whole, which nothing promises for two 32-bit elements side by side (the PTX memory model
takes a vector access as one access of each element).  No run shows the difference, so the source is
read: tag_store and tag_load take the tag and its half as one element."""
import os
import re

from eig_gb300 import build as B


def test_tag_and_half_are_one_element():
    text = open(os.path.join(B.CSRC, "gp_eig.cu")).read()
    for name, op in (("tag_store", "st"), ("tag_load", "ld")):
        body = text.split(name + "(", 1)[1].split("\n}\n", 1)[0]
        assert re.findall(r"%s\.relaxed[\w.]*" % op, body) == [op + ".relaxed.gpu.global.v2.b64"]
