// The kernels of an order P = p + 1 are translation units of their own
// (build.py compiles the files that have them once with DGB_ORDER = 1..7 for
// the kernels and once without it for the dispatch): the driver loads a unit
// as a whole, its line tables with it, when its first kernel is launched, and a
// handle launches one order.  Handle, step, residual,
// product, recorded run and gradient on a fresh context, all orders in a unit
// against one: 96 -> 36 ms at 12^3 p = 4, 96 -> 34 at 16^3 p = 3, 93 -> 22 on
// curved elements with heat flux at p = 2 (10^3).
#pragma once

#define DGB_EACH_ORDER(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7)
