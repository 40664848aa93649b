"""The library's translation units share the namespace olv: a type defined in two of
them would be two types of one name (CPU check of the sources)."""
import collections
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_types_are_defined_once():
    where = collections.defaultdict(set)
    for path in glob.glob(os.path.join(ROOT, "olive_b200", "csrc", "*.cu*")):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        text = re.sub(r"namespace \{.*?^\}  *$", "", text, flags=re.S | re.M)
        for name in re.findall(r"^(?:struct|class|union)(?: alignas\(\d+\))? (\w+)[^;{]*\{", text,
                               flags=re.M):
            where[name].add(os.path.basename(path))
    assert len(where) > 40
    assert not {n: sorted(f) for n, f in where.items() if len(f) > 1}
