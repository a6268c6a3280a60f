"""Batches that reach each form of the time loops, by sweep: (approximation,
boundary, sweep, rows per thread, (nz, nx, border, shots)).  The tests assert
that they do."""

TILES = [
    ("acoustic", "cerjan", "forward", 2, (61, 133, 12, 2)), ("acoustic", "cerjan", "forward", 3, (16, 38, 8, 40)),
    ("acoustic", "cerjan", "forward", 4, (91, 48, 10, 40)), ("VTI", "cerjan", "forward", 2, (49, 111, 10, 3)),
    ("VTI", "cerjan", "forward", 3, (44, 84, 8, 30)), ("VTI", "cerjan", "forward", 4, (18, 41, 8, 97)),
    ("TTI", "cerjan", "forward", 2, (95, 52, 8, 40)), ("TTI", "cerjan", "forward", 3, (27, 22, 8, 64)),
    ("TTI", "cerjan", "forward", 4, (18, 41, 8, 97)), ("acoustic", "CPML", "forward", 1, (40, 60, 10, 12)),
    ("VTI", "CPML", "forward", 1, (43, 63, 9, 12)), ("acoustic", "CPML", "forward", 1, (287, 653, 45, 1)),
    ("VTI", "CPML", "forward", 1, (287, 653, 45, 1)),
    ("acoustic", "cerjan", "exact", 2, (61, 133, 12, 2)), ("acoustic", "cerjan", "exact", 3, (84, 32, 8, 16)),
    ("acoustic", "cerjan", "exact", 4, (16, 25, 8, 161)), ("acoustic", "cerjan", "exact", 4, (215, 148, 10, 40)),
    ("acoustic", "cerjan", "rtm", 2, (61, 133, 12, 2)), ("acoustic", "cerjan", "rtm", 3, (123, 16, 8, 45)),
    ("acoustic", "cerjan", "rtm", 4, (16, 25, 8, 161)), ("acoustic", "CPML", "rtm", 1, (43, 63, 9, 12)),
    ("acoustic", "cerjan", "reverse", 2, (61, 133, 12, 2)), ("acoustic", "cerjan", "reverse", 3, (80, 180, 10, 16)),
    ("acoustic", "cerjan", "reverse", 4, (92, 92, 8, 100)), ("VTI", "cerjan", "reverse", 2, (61, 133, 12, 2)),
    ("VTI", "cerjan", "reverse", 3, (80, 180, 10, 16)), ("VTI", "cerjan", "reverse", 4, (16, 16, 8, 100)),
    ("TTI", "cerjan", "reverse", 2, (16, 16, 8, 100)), ("TTI", "cerjan", "reverse", 3, (12, 87, 8, 100)),
    ("TTI", "cerjan", "reverse", 4, (116, 383, 10, 16)),
]

# one cooperative launch with a barrier after every step
PERSISTENT = [("acoustic", (933, 959, 20, 1)), ("VTI", (197, 377, 20, 8)), ("TTI", (250, 89, 20, 16)),
              ("TTI", (451, 1101, 50, 1))]


def ident(v):
    return "-".join("x".join(map(str, x)) if isinstance(x, tuple) else str(x) for x in v)
