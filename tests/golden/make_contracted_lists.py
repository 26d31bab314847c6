"""Digests of the contracted flavour's lists, from a build of the first
revision of this repository's engine whose contraction nvcc chose (the
revisions before "Tetrahedron enumeration decides candidates by a certified
pencil filter"), on the inputs of tests/test_contraction.py:

    python tests/golden/make_contracted_lists.py <built tree of that revision>

writes tests/golden/contracted_lists.json (needs a GPU).  The as-run digests
were taken once from the same build, on inputs where its counting and its
writing pass agreed: where they do not, it writes past its list, so it is not
run in that mode here."""
import importlib.util
import json
import os
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path[:0] = [os.path.dirname(HERE), os.path.dirname(os.path.dirname(HERE))]


def main():
    pkg = os.path.join(sys.argv[1], "parallelac-xmp_b200")
    spec = importlib.util.spec_from_file_location("parallelac_xmp_b200", os.path.join(pkg, "__init__.py"),
                                                  submodule_search_locations=[pkg])
    pac = importlib.util.module_from_spec(spec)
    sys.modules["parallelac_xmp_b200"] = pac
    spec.loader.exec_module(pac)
    import test_contraction as tc
    path = sys.argv[2] if len(sys.argv) > 2 else os.path.join(HERE, "contracted_lists.json")
    out = {k: v for k, v in json.load(open(path)).items() if k.startswith("as-run")} if os.path.exists(path) else {}
    for name in tc.AS_WRITTEN:
        out[name] = tc.record(pac, name)
        print(name, out[name]["counts"], flush=True)
    with open(path, "w") as f:
        json.dump(out, f, indent=1, sort_keys=True)


if __name__ == "__main__":
    main()
