"""The kernels of a pass are launched with programmatic serialisation: a kernel is alive while the one
before it writes.  The read-only path (CR_LDG, restricted pointers) is defined for data that does not
change in a kernel's life, so in the bodies of those kernels it may only take what a solve leaves alone."""
import os
import re

BODY = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "copsandrobbers_gb300", "csrc", "crgpu_v1_body.cuh")
# the graph, its masks and lists, the rank table, the configurations
FIXED = {"B", "binom", "configs", "rp", "adj", "rrp", "radj", "nbr", "iso", "isolated", "hop", "h", "cover",
         "cin", "ell", "ell_off"}
WRITTEN = ("front", "fflag", "list", "clist", "h1", "cand", "cbits", "marked", "table", "meta", "sync")


def code():
    return re.sub(r"//[^\n]*", "", open(BODY).read())


def test_read_only_loads_take_fixed_data_only():
    names = set()
    for arg in re.findall(r"CR_LDG\(([^;]*)", code()):
        arg = re.sub(r"^(reinterpret_cast<[^>]*>\(|&)+", "", arg)
        names.add(re.match(r"(?:d\.(?:g\.)?)?(\w+)", arg).group(1))
    names.discard("p")   # Cov8::load's argument, a row of the cover masks
    assert names <= FIXED, sorted(names - FIXED)


def test_a_load_helper_of_the_read_only_path_has_fixed_callers():
    # the one helper that takes an address: Cov8::load
    helpers = re.findall(r"__device__ __forceinline__ void (\w+)\(const (\w+)\* p\) \{[^}]*CR_LDG", code())
    assert helpers == [("load", "uint8_t")], helpers
    assert all("cover" in a or a == "cv" for a in re.findall(r"\b(?:t|z)\.load\(([^;]*)\);", code()))


def test_restricted_pointers_point_at_fixed_data():
    bound = re.findall(r"CR_RESTRICT (\w+) = ([^;]*);", code())
    assert bound
    for name, value in bound:
        assert not any(re.search(rf"\bd\.{w}\b", value) for w in WRITTEN), (name, value)
