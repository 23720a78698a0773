"""Domains whose interface solves take each route of the solve plans, shared by
the CPU and GPU tests of those."""
from hierarchicaldd_b200 import domains

ROUTES = ["one tree", "pairs", "quads", "fronts in pairs", "slots in memory", "cut factors",
          "equal cut factors", "ragged", "forest"]


def domain(name):
    """(domain, sigma levels) of a route."""
    if name == "one tree":              # interface systems of a few hundred unknowns: one CTA
        return domains.small(16, 8, 3, seed=4), 2
    if name == "pairs":                 # 2 trees per CTA
        return domains.small((40, 36, 44), 8, 6, seed=4), 2
    if name == "quads":                 # 4 trees per CTA
        return domains.small((56, 56, 64), 8, 6, seed=4), 2
    if name == "fronts in pairs":       # 2 trees per CTA; cut interface systems
        return domains.small(96, 16, 20, seed=4), 3
    if name == "slots in memory":       # 32^3 interiors: update slots do not fit
        return domains.small(128, 32, 24, seed=4), 2
    if name == "cut factors":           # few large trees: cut
        return domains.small(64, 32, 9, seed=4), 2
    if name == "equal cut factors":     # ... most of them with the same factor
        return domains.small((96, 64, 64), 32, 0, seed=4), 2
    if name == "ragged":
        return domains.small((33, 40, 41), 16, 5, seed=4), 2
    # Many components: plans of thousands of tiny fronts, trees without fronts above.
    d = domains.config5(16)
    d.meta.update(vlevels=3, interior_smoothing=3, boundary_smoothing=3)
    return domains.Domain(d.size, d.flags, d.rhs, (8, 8, 8), d.name, d.meta), 2
