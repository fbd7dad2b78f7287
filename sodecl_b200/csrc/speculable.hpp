// Whether a system file may run on numbers that its own functions never gave.
#pragma once

#include <string>

namespace sodecl_b200 {

// The speculative copy of a system file (device/fastmath.cuh) computes a step
// whose result is thrown away when an argument turns out to lie outside the
// range of a straight-line function or quotient.  Until then the file's own
// code goes on with a number that the plain file would not have seen there.
// That is harmless for arithmetic; it is not where numbers decide how long a
// loop runs or which address is read.  Empty when `code` (comments blanked)
// keeps the two apart, else the first thing found that does not:
//  - loops other than `for` over an int with bounds and step of ints;
//  - ints that get their value from anything but int literals, the program's
//    sizes, other such ints, or a comparison (0 or 1, and then not used in a
//    subscript, a bound or as an int argument): conversions, arrays of ints,
//    functions that return them, assignments outside a for's header;
//  - subscripts of anything but such ints; pointers other than parameters, and
//    parameters that are moved; recursion, and functions as values;
//  - and what the scan below does not follow: goto, switch, #include, type
//    definitions, templates, inline assembly, printf.
// The scan is of tokens, not of a syntax tree: it refuses some files that would
// be safe (they are built without the speculative copy), and every conversion
// to an integer type needs one of the forms above to be accepted.
std::string speculation_hazard(const std::string &code);

}  // namespace sodecl_b200
