// What a bulk copy moves of a chunk of doubles (plain C++, also compiled by the host tests).
#pragma once

#ifdef __CUDACC__
#define PFG_HD __host__ __device__ __forceinline__
#else
#define PFG_HD inline
#endif

namespace pfg
{

// A bulk copy moves whole 16-byte units.  Values v0 .. v0 + nv of an array of n doubles (nv 0:
// none), the first at an address that is odd modulo 16 bytes (odd: 8 behind a boundary): the
// copy takes entries [begin, end), counted from v0, rounded out to the units where these lie
// in the array; lo / hi: the first / last value has to be loaded by itself, because its unit
// reaches past the array's start / end (a caller's array may begin on 8 bytes, and nnz be odd).
struct BulkSpan
{
	int begin, end;
	bool lo, hi;
};
PFG_HD BulkSpan bulk_span(int v0, int nv, int n, int odd)
{
	BulkSpan s = {0, 0, false, false};
	if (nv <= 0) return s;
	s.begin = -odd;
	s.end = nv + ((nv + odd) & 1);
	if (v0 + s.begin < 0)
	{
		s.begin += 2;
		s.lo = true;
	}
	if ((long long)v0 + s.end > n)
	{
		s.end -= 2;
		s.hi = true;
	}
	if (s.end < s.begin) s.end = s.begin;
	return s;
}

} // namespace pfg
